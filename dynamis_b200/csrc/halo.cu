// Partition bookkeeping and halo-map assembly for B200 (sm_100a).
//
//   dynb_bincount_i64 / dynb_select_eq_i64   atom_counts and partition_indices of
//       SFCPartitioner::do_partition (dynamis_state/src/csrc/partition/sfc_partitioner.cpp:166-176)
//   dynb_halo_mark_from_edges                per-edge pass of extract_halo_info
//       (dynamis_state/src/csrc/graph/dist_graph_ops_kernels.cu:46-59, 104-188)
//   dynb_halo_lists_plan / _fill             send and recv CSR of build_halo_maps
//       (dynamis_state/src/csrc/build_halo_maps.cpp:60-125) and of extract_halo_info, from
//       per-atom rank bit masks instead of the reference's [N, W] bool matrix + nonzero + argsort
//   dynb_csr_plan / dynb_csr_fill            one such list per call, from one mask
//   dynb_filter_edges_plan / _fill           filter_edges_to_radius
//       (dist_graph_ops_kernels.cu:16-43, 62-102)
//
// Every list these produce is in the reference's order: grouped by peer rank ascending, inside a
// peer ascending atom id.  That order falls out of a stable per-peer compaction over atoms in
// ascending id, so nothing is sorted.

#include "common.cuh"
#include "clear.cuh"
#include "scan.cuh"

namespace dynb {

// ------------------------------------------------------------------------------------------ bincount / select
__global__ void __launch_bounds__(256)
bincount_i64_kernel(const int64_t* a, int64_t n, int64_t W, unsigned long long* counts,
                    uint32_t* bad)
{
    chain_begin();
    extern __shared__ uint32_t hist[];
    const bool use_smem = W <= 4096;
    if (use_smem) {
        for (int k = threadIdx.x; k < W; k += blockDim.x) hist[k] = 0;
        __syncthreads();
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = a[i];
        if (v < 0 || v >= W) { atomicOr(bad, 1u); continue; }
        if (use_smem) atomicAdd(&hist[v], 1u);
        else atomicAdd(&counts[v], 1ull);
    }
    if (use_smem) {
        __syncthreads();
        for (int k = threadIdx.x; k < W; k += blockDim.x)
            if (hist[k]) atomicAdd(&counts[k], (unsigned long long)hist[k]);
    }
}

// Stream compaction in two launches: matches per tile, then every block adds up the tiles in front of its own and writes its
// matches.  A warp owns 256 consecutive values, so that the order is kept by ballots alone.  Adding up is quadratic in the
// tiles: above SELECT_FUSED_MAX_TILES (16.8 M values) a prefix sum over the tiles goes between the two (40 M values 160 us
// either way, 100 M 296 against 412 us without it, 10^9 2.4 against 24.7 ms; a flag and a prefix sum per value took 10.0 ms).
constexpr int SELECT_TILE = 2048;
constexpr int64_t SELECT_FUSED_MAX_TILES = 8192;

__global__ void __launch_bounds__(256)
select_count_kernel(const int64_t* a, int64_t n, int64_t value, uint32_t* tile_count)
{
    chain_begin();
    __shared__ uint32_t wsum[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * SELECT_TILE + warp * 256 + lane;
    int64_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = (base + 32 * k < n) ? a[base + 32 * k] : ~value;
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) c += (v[k] == value) ? 1u : 0u;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) wsum[warp] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t s = 0;
        for (int w = 0; w < 8; w++) s += wsum[w];
        tile_count[blockIdx.x] = s;
    }
}

template <bool SUMMED>   // tile_count holds the matches in front of each tile already
__global__ void __launch_bounds__(256)
select_fill_kernel(const int64_t* a, int64_t n, int64_t value, const uint32_t* tile_count,
                   const int64_t* gather_src, int64_t* out, int64_t* count_out)
{
    chain_begin();
    __shared__ uint32_t wsum[8], before[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * SELECT_TILE + warp * 256 + lane;
    int64_t v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = (base + 32 * k < n) ? a[base + 32 * k] : ~value;
    uint32_t s = 0;
    if (!SUMMED) {
        for (int i = threadIdx.x; i < (int)blockIdx.x; i += 256) s += tile_count[i];
        s = __reduce_add_sync(0xffffffffu, s);
    } else if (threadIdx.x == 0) {
        s = tile_count[blockIdx.x];
    }
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) c += (v[k] == value) ? 1u : 0u;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) { before[warp] = s; wsum[warp] = c; }
    __syncthreads();
    uint32_t at = 0;
    for (int w = 0; w < 8; w++) at += before[w];
    if (!SUMMED && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *count_out = (int64_t)at + tile_count[blockIdx.x];
    for (int w = 0; w < warp; w++) at += wsum[w];
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint32_t m = __ballot_sync(0xffffffffu, v[k] == value);
        if (v[k] == value) {
            const int64_t i = base + 32 * k;
            out[at + __popc(m & lt)] = gather_src ? gather_src[i] : i;
        }
        at += __popc(m);
    }
}


// ------------------------------------------------------------------------------------------ edge marking
// For every edge src -> dst of one rank's edge list (dst owned by my_rank): when the source is
// owned by a peer p, that peer must send src to me (recv side) and I must send dst to p (send
// side, by the symmetry of the radius graph).
// Four edges a thread: bound by the latency of an edge's ends and then its owner, which are in flight for all four (5.6 M edges, one edge
// a thread: 40 us with what it waits for, four 36).
constexpr int MARK_EDGES = 4;
__global__ void __launch_bounds__(256)
halo_mark_edges_kernel(const int64_t* src, const int64_t* dst, int64_t E,
                       const int64_t* pid, int64_t N, int64_t my_rank, int words,
                       uint32_t* send_mask, uint32_t* recv_mask,
                       uint8_t* has_remote, uint32_t* bad)
{
    chain_begin();
    const int64_t e0 = (int64_t)blockIdx.x * (MARK_EDGES * 256) + threadIdx.x;
    int64_t s[MARK_EDGES], d[MARK_EDGES], owner[MARK_EDGES];
#pragma unroll
    for (int k = 0; k < MARK_EDGES; k++) {
        const bool in = e0 + 256 * k < E;
        s[k] = in ? src[e0 + 256 * k] : 0;
        d[k] = in ? dst[e0 + 256 * k] : 0;
    }
    // my_rank: nothing to do
    uint32_t wrong = 0u;
#pragma unroll
    for (int k = 0; k < MARK_EDGES; k++) {
        owner[k] = my_rank;
        if (e0 + 256 * k >= E) continue;
        if (s[k] < 0 || s[k] >= N || d[k] < 0 || d[k] >= N) wrong |= 1u;
        else owner[k] = pid[s[k]];
    }
#pragma unroll
    for (int k = 0; k < MARK_EDGES; k++) {
        const int64_t p = owner[k];
        if (p == my_rank) continue;
        if (p < 0 || p >= (int64_t)words * 32) { wrong |= 2u; continue; }
        const uint32_t bit = 1u << (p & 31);
        uint32_t* rw = &recv_mask[s[k] * words + (p >> 5)];
        if (!(*rw & bit)) atomicOr(rw, bit);
        uint32_t* sw = &send_mask[d[k] * words + (p >> 5)];
        if (!(*sw & bit)) atomicOr(sw, bit);
        has_remote[d[k]] = 1;
    }
    if (wrong) atomicOr(bad, wrong);
}

// ------------------------------------------------------------------------------------------ halo lists
// Atom a in [0, n) carries two sets of peer ranks, S(a) and R(a).  Send segment p lists the atoms with p in S(a), recv
// segment p those with p in R(a), each ascending in a.  Either the sets are given as bit masks (extract_halo_info), or
// they follow from one "needed by" mask and the owners (build_halo_maps):
//   S(a) = owner[a] == me ? ranks that need a, without me : {}
//   R(a) = owner[a] != me and I need a ? {owner[a]} : {}
// and the own atoms themselves (owner[a] == me, ascending) give the local indices.  Peers are ranks below W: an owner or a
// mask bit beyond them is in no set, in the counting and in the writing pass alike.
//
// Both lists, the local indices and the interior mask come out of one counting and one writing pass over the masks; most
// atoms have empty sets, so a warp (128 consecutive atoms, 32 at a time) works on the peers that occur and on no others.
// One million atoms, 8 ranks: 9 + 10 + 18 us (count, row scan, fill), where per-list passes that walked all peers took 120.
constexpr int HL_THREADS = 256;
constexpr int HL_WARPS = HL_THREADS / 32;
constexpr int HL_ROUNDS = 4;
constexpr int HL_TILE = HL_THREADS * HL_ROUNDS;

struct HaloSets {
    const uint32_t* send_mask;   // masks of S(a), or of "needed by" when owner != nullptr
    const uint32_t* recv_mask;   // masks of R(a); not read when owner != nullptr
    const int64_t* owner;
    int64_t n, me;
    int words, W;
};

// the sets of this lane's HL_ROUNDS atoms (base, base + 32, ...) among the 32 peers of one mask word; all loads first
__device__ __forceinline__ void halo_sets(const HaloSets& h, int64_t base, int word, uint32_t (&s)[HL_ROUNDS], uint32_t (&r)[HL_ROUNDS],
                                          uint32_t& own)
{
    uint32_t mw[HL_ROUNDS], mr[HL_ROUNDS];
    int64_t o[HL_ROUNDS];
    const bool owners = h.owner != nullptr;
    const uint32_t* second = owners ? h.send_mask + (h.me >> 5) : h.recv_mask + word;
#pragma unroll
    for (int k = 0; k < HL_ROUNDS; k++) {
        const int64_t a = base + 32 * k;
        const bool live = a < h.n;
        mw[k] = live ? h.send_mask[a * h.words + word] : 0u;
        mr[k] = live ? second[a * h.words] : 0u;
        o[k] = (live && owners) ? h.owner[a] : -1;
    }
    own = 0u;
    const uint32_t peers = h.W - 32 * word < 32 ? (1u << (h.W - 32 * word)) - 1u : ~0u;
#pragma unroll
    for (int k = 0; k < HL_ROUNDS; k++) {
        s[k] = mw[k];
        r[k] = mr[k];
        if (owners) {
            const bool mine = o[k] == h.me;
            if (mine) own |= 1u << k;
            s[k] = !mine ? 0u : (word == (int)(h.me >> 5) ? mw[k] & ~(1u << (h.me & 31)) : mw[k]);
            r[k] = (!mine && (o[k] >> 5) == word && ((mr[k] >> (h.me & 31)) & 1u)) ? 1u << (o[k] & 31) : 0u;
        }
        s[k] &= peers;
        r[k] &= peers;
    }
}

// lane p of the warp adds up how many of the 32 sets contain p
__device__ __forceinline__ uint32_t halo_count_sets(uint32_t set, int lane)
{
    uint32_t c = 0;
    for (uint32_t any = __reduce_or_sync(0xffffffffu, set); any; any &= any - 1) {
        const int p = __ffs((int)any) - 1;
        const uint32_t m = __ballot_sync(0xffffffffu, (set >> p) & 1u);
        if (lane == p) c = __popc(m);
    }
    return c;
}

// rows of bsum (nblocks entries each): send peers 0..W-1, recv peers 0..W-1, own atoms
__global__ void __launch_bounds__(HL_THREADS)
halo_lists_count_kernel(const HaloSets h, int W, int nblocks, uint32_t* bsum)
{
    chain_begin();
    __shared__ uint32_t ws[HL_WARPS][2][32];
    __shared__ uint32_t wown[HL_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * HL_TILE + warp * 32 * HL_ROUNDS + lane;
    for (int word = 0; word < h.words; word++) {
        uint32_t s[HL_ROUNDS], r[HL_ROUNDS], own, cs = 0, cr = 0;
        halo_sets(h, base, word, s, r, own);
#pragma unroll
        for (int k = 0; k < HL_ROUNDS; k++) {
            cs += halo_count_sets(s[k], lane);
            cr += halo_count_sets(r[k], lane);
        }
        const uint32_t co = __reduce_add_sync(0xffffffffu, __popc(own));
        __syncthreads();
        ws[warp][0][lane] = cs;
        ws[warp][1][lane] = cr;
        if (lane == 0) wown[warp] = co;
        __syncthreads();
        if (threadIdx.x < 64) {
            const int which = threadIdx.x >> 5, p = word * 32 + lane;
            uint32_t t = 0;
            for (int w = 0; w < HL_WARPS; w++) t += ws[w][which][lane];
            if (p < W) bsum[(int64_t)(which * W + p) * nblocks + blockIdx.x] = t;
        } else if (threadIdx.x == 64 && word == 0) {
            uint32_t t = 0;
            for (int w = 0; w < HL_WARPS; w++) t += wown[w];
            bsum[(int64_t)(2 * W) * nblocks + blockIdx.x] = t;
        }
    }
}

// One block per row: exclusive scan of the row of block sums (in place) and its total; the block that finishes last turns
// the totals into offsets [send W + 1 | recv W + 1 | number of own atoms].
__global__ void __launch_bounds__(SCAN_THREADS)
halo_lists_scan_kernel(uint32_t* bsum, int nblocks, int W, int64_t* totals, uint32_t* arrived,
                       int64_t* offsets, int64_t* words_host, int n_words)
{
    chain_begin();
    __shared__ uint32_t warp_sums[SCAN_THREADS / 32];
    __shared__ bool last;
    uint32_t* row = bsum + (int64_t)blockIdx.x * nblocks;
    uint32_t carry = 0;
    for (int b0 = 0; b0 < nblocks; b0 += SCAN_THREADS * 4) {
        const int i = b0 + threadIdx.x * 4;
        uint32_t v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) { v[k] = (i + k < nblocks) ? row[i + k] : 0u; sum += v[k]; }
        uint32_t tot;
        uint32_t run = carry + block_excl_scan<uint32_t>(sum, &tot, warp_sums);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i + k < nblocks) row[i + k] = run;
            run += v[k];
        }
        carry += tot;
    }
    if (threadIdx.x == 0) {
        totals[blockIdx.x] = (int64_t)carry;
        __threadfence();
        last = atomicAdd(arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    if (threadIdx.x == 0) {
        __threadfence();
        for (int which = 0; which < 2; which++) {
            int64_t run = 0;
            for (int p = 0; p < W; p++) {
                offsets[which * (W + 1) + p] = run;
                run += __ldcg(reinterpret_cast<const long long*>(totals) + which * W + p);
            }
            offsets[which * (W + 1) + W] = run;
        }
        offsets[2 * (W + 1)] = __ldcg(reinterpret_cast<const long long*>(totals) + 2 * W);
    }
    // to the caller's pinned memory from here: a copy behind this launch is one of another engine, 10 us
    if (words_host == nullptr) return;
    __syncthreads();
    for (int i = threadIdx.x; i < n_words; i += blockDim.x) words_host[i] = __ldcg(reinterpret_cast<const long long*>(offsets) + i);
}

struct HaloListsOut {
    const int64_t* value_map;    // send list entry of atom a when the owners are not given (global -> local)
    const uint8_t* has_foreign;  // by atom; with the owners given
    int64_t* send_local;
    int64_t* recv_atom;
    int64_t* recv_ghost;
    uint8_t* interior;           // by local index; with the owners given
    int64_t* matrix_row;         // [W] rows sent to every rank, n_local at the own place; or nullptr
    int64_t n_local;
};

__global__ void __launch_bounds__(HL_THREADS)
halo_lists_fill_kernel(const HaloSets h, int W, int nblocks, const uint32_t* bsum, const int64_t* offsets,
                       const HaloListsOut out)
{
    chain_begin();
    __shared__ uint32_t ws[HL_WARPS][2][32];
    __shared__ uint32_t wown[HL_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = lanemask_lt();
    const int64_t base = (int64_t)blockIdx.x * HL_TILE + warp * 32 * HL_ROUNDS + lane;
    if (blockIdx.x == 0 && out.matrix_row != nullptr)
        for (int p = threadIdx.x; p < W; p += HL_THREADS) out.matrix_row[p] = p == (int)h.me ? out.n_local : offsets[p + 1] - offsets[p];
    for (int word = 0; word < h.words; word++) {
        uint32_t set[2][HL_ROUNDS], mine_own, own[HL_ROUNDS], c[2] = {0u, 0u}, co = 0;
        halo_sets(h, base, word, set[0], set[1], mine_own);
#pragma unroll
        for (int k = 0; k < HL_ROUNDS; k++) {
            own[k] = __ballot_sync(0xffffffffu, (mine_own >> k) & 1u);
            c[0] += halo_count_sets(set[0][k], lane);
            c[1] += halo_count_sets(set[1][k], lane);
            co += __popc(own[k]);
        }
        __syncthreads();
        ws[warp][0][lane] = c[0];
        ws[warp][1][lane] = c[1];
        if (lane == 0) wown[warp] = co;
        __syncthreads();
        // lane p: place of this warp's first entry in segment p of the send and of the recv list
        const int p = word * 32 + lane;
        int64_t at[2] = {0, 0};
        if (p < W) {
#pragma unroll
            for (int which = 0; which < 2; which++) {
                at[which] = offsets[which * (W + 1) + p] + bsum[(int64_t)(which * W + p) * nblocks + blockIdx.x];
                for (int w = 0; w < warp; w++) at[which] += ws[w][which][lane];
            }
        }
        int64_t first_own = 0;
        if (h.owner != nullptr) {
            first_own = bsum[(int64_t)(2 * W) * nblocks + blockIdx.x];
            for (int w = 0; w < warp; w++) first_own += wown[w];
        }
#pragma unroll
        for (int k = 0; k < HL_ROUNDS; k++) {
            const int64_t a = base + 32 * k;
            const int64_t local = first_own + __popc(own[k] & lt);
            if (word == 0 && ((own[k] >> lane) & 1u)) out.interior[local] = out.has_foreign[a] ? 0 : 1;
            first_own += __popc(own[k]);
#pragma unroll
            for (int which = 0; which < 2; which++) {
                const uint32_t mine = set[which][k];
                for (uint32_t any = __reduce_or_sync(0xffffffffu, mine); any; any &= any - 1) {
                    const int q = __ffs((int)any) - 1;
                    const uint32_t m = __ballot_sync(0xffffffffu, (mine >> q) & 1u);
                    const int64_t e = __shfl_sync(0xffffffffu, (long long)at[which], q) + __popc(m & lt);
                    if ((mine >> q) & 1u) {
                        if (which == 0) {
                            out.send_local[e] = h.owner != nullptr ? local : out.value_map[a];
                        } else {
                            out.recv_atom[e] = a;
                            out.recv_ghost[e] = out.n_local + e;
                        }
                    }
                    if (lane == q) at[which] += __popc(m);
                }
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------ CSR assembly
// Element a in [0, n) carries a set of peer ranks.  For each peer p, the output segment p lists the
// elements whose set contains p, ascending in a.  One list per call, every peer walked: the form for C callers that have
// one mask at a time; the partitioner's and extract_halo_info's two lists come from the halo list passes above.  Modes
// define the set:
enum { CSR_SEND = 0, CSR_RECV = 1, CSR_RAW = 2 };
//   CSR_SEND  owner[a] == R ? bits of mask[a] without R : {}        (needed_by rows of my atoms)
//   CSR_RECV  owner[a] != R and bit R of mask[a] ? {owner[a]} : {}   (foreign atoms I need)
//   CSR_RAW   bits of mask[a]
constexpr int CSR_THREADS = 256;
constexpr int CSR_WARPS = CSR_THREADS / 32;

__device__ __forceinline__ bool csr_has(const uint32_t* __restrict__ mask, int words, const int64_t* __restrict__ owner,
                                        int64_t a, int64_t R, int mode, int p)
{
    if (mode == CSR_RAW) return (mask[a * words + (p >> 5)] >> (p & 31)) & 1u;
    const int64_t o = owner[a];
    if (mode == CSR_SEND) return o == R && p != R && ((mask[a * words + (p >> 5)] >> (p & 31)) & 1u);
    return o != R && o == p && ((mask[a * words + (R >> 5)] >> (R & 31)) & 1u);
}

// bsum[p * nblocks + block] = number of elements of this block whose set contains p
__global__ void __launch_bounds__(CSR_THREADS)
csr_count_kernel(const uint32_t* __restrict__ mask, int words, const int64_t* __restrict__ owner, int64_t n, int64_t R,
                 int mode, int W, int nblocks, uint32_t* __restrict__ bsum)
{
    __shared__ uint32_t wsum[CSR_WARPS];
    const int64_t a = (int64_t)blockIdx.x * CSR_THREADS + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int p = 0; p < W; p++) {
        const bool f = (a < n) && csr_has(mask, words, owner, a, R, mode, p);
        const uint32_t b = __ballot_sync(0xffffffffu, f);
        if (lane == 0) wsum[warp] = __popc(b);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t s = 0;
            for (int w = 0; w < CSR_WARPS; w++) s += wsum[w];
            bsum[(int64_t)p * nblocks + blockIdx.x] = s;
        }
        __syncthreads();
    }
}

// One block per peer: exclusive scan of its row of block sums (in place) and the row total.
__global__ void __launch_bounds__(SCAN_THREADS)
csr_scan_rows_kernel(uint32_t* __restrict__ bsum, int nblocks, int64_t* __restrict__ totals)
{
    __shared__ uint32_t warp_sums[SCAN_THREADS / 32];
    uint32_t* row = bsum + (int64_t)blockIdx.x * nblocks;
    uint32_t carry = 0;
    for (int b0 = 0; b0 < nblocks; b0 += SCAN_THREADS) {
        const int i = b0 + threadIdx.x;
        const uint32_t v = (i < nblocks) ? row[i] : 0u;
        uint32_t tot;
        const uint32_t ex = block_excl_scan<uint32_t>(v, &tot, warp_sums);
        if (i < nblocks) row[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = (int64_t)carry;
}

__global__ void csr_offsets_kernel(const int64_t* __restrict__ totals, int W, int64_t* __restrict__ offsets)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        int64_t run = 0;
        for (int p = 0; p < W; p++) { offsets[p] = run; run += totals[p]; }
        offsets[W] = run;
    }
}

__global__ void __launch_bounds__(CSR_THREADS)
csr_fill_kernel(const uint32_t* __restrict__ mask, int words, const int64_t* __restrict__ owner, int64_t n, int64_t R,
                int mode, int W, int nblocks, const uint32_t* __restrict__ bsum, const int64_t* __restrict__ offsets,
                const int64_t* __restrict__ value_map, int64_t* __restrict__ out)
{
    __shared__ uint32_t wsum[CSR_WARPS];
    const int64_t a = (int64_t)blockIdx.x * CSR_THREADS + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = lanemask_lt();
    for (int p = 0; p < W; p++) {
        const bool f = (a < n) && csr_has(mask, words, owner, a, R, mode, p);
        const uint32_t b = __ballot_sync(0xffffffffu, f);
        if (lane == 0) wsum[warp] = __popc(b);
        __syncthreads();
        if (f) {
            uint32_t before = 0;
            for (int w = 0; w < warp; w++) before += wsum[w];
            const int64_t pos = offsets[p] + bsum[(int64_t)p * nblocks + blockIdx.x] + before + __popc(b & lt);
            out[pos] = value_map ? value_map[a] : a;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256)
gather_not_u8_kernel(const uint8_t* flags, const int64_t* idx, int64_t n, uint8_t* out)
{
    chain_begin();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = flags[idx[i]] ? 0 : 1;
}

__global__ void __launch_bounds__(256)
scatter_iota_kernel(const int64_t* idx, int64_t n, int64_t N, int64_t* g2l, uint32_t* bad)
{
    chain_begin();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t a = idx[i];
    if (a < 0 || a >= N) { atomicOr(bad, 4u); return; }
    g2l[a] = i;
}

// ------------------------------------------------------------------------------------------ edge filter
// keep[e] = |pos[src] + shift @ cell - pos[dst]|^2 <= r2, float32, the reference's expression
// (dist_graph_ops_kernels.cu:30-43).
struct Cell9 { float c[9]; };

// Edge filter.  A block tests FILTER_TILE edges, keeps one bit per edge and counts the tile; a prefix sum over the tiles'
// counts gives every tile its place and the second pass finds an edge's place inside the tile from the bits.  Bound by
// reading the edges twice and writing the kept ones (56 + 28 bytes an edge).  A 32-bit flag per edge and a prefix sum over
// all edges (5.6 M: 46 us flags, 32 us prefix sum, 53 us compaction) cost the refresh of 250 k atoms 24 us more.
constexpr int FILTER_ROUNDS = 4;                       // edges per thread, in flight together
constexpr int FILTER_TILE = 256 * FILTER_ROUNDS;       // 32 words of 32 edges
static_assert(FILTER_TILE == 1024, "a warp reads a tile's words in one load");

__global__ void __launch_bounds__(256)
edge_keep_bits_kernel(const int64_t* src, const int64_t* dst, const float* shifts,
                      const float* pos, Cell9 cell, float r2, int64_t E, uint32_t* bits,
                      uint32_t* tile_count)
{
    chain_begin();
    __shared__ uint32_t warp_count[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t e0 = (int64_t)blockIdx.x * FILTER_TILE + threadIdx.x;
    int64_t s[FILTER_ROUNDS], d[FILTER_ROUNDS];
    float h[FILTER_ROUNDS][3];
#pragma unroll
    for (int k = 0; k < FILTER_ROUNDS; k++) {
        const int64_t e = e0 + 256 * k;
        const bool in = e < E;
        s[k] = in ? src[e] : 0;
        d[k] = in ? dst[e] : 0;
#pragma unroll
        for (int c = 0; c < 3; c++) h[k][c] = in ? shifts[3 * e + c] : 0.0f;
    }
    uint32_t count = 0;
#pragma unroll
    for (int k = 0; k < FILTER_ROUNDS; k++) {
        bool keep = false;
        if (e0 + 256 * k < E) {
            float sx = pos[3 * s[k] + 0], sy = pos[3 * s[k] + 1], sz = pos[3 * s[k] + 2];
            const float dx = pos[3 * d[k] + 0], dy = pos[3 * d[k] + 1], dz = pos[3 * d[k] + 2];
            const float h0 = h[k][0], h1 = h[k][1], h2 = h[k][2];
            sx += h0 * cell.c[0] + h1 * cell.c[3] + h2 * cell.c[6];
            sy += h0 * cell.c[1] + h1 * cell.c[4] + h2 * cell.c[7];
            sz += h0 * cell.c[2] + h1 * cell.c[5] + h2 * cell.c[8];
            const float ax = sx - dx, ay = sy - dy, az = sz - dz;
            keep = (ax * ax + ay * ay + az * az) <= r2;
        }
        const uint32_t word = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) bits[(int64_t)blockIdx.x * 32 + 8 * k + warp] = word;
        count += __popc(word);
    }
    if (lane == 0) warp_count[warp] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) total += warp_count[w];
        tile_count[blockIdx.x] = total;
    }
}

__global__ void __launch_bounds__(256)
edge_compact_kernel(const int64_t* edges, const unsigned char* shifts_raw, int shift_row_bytes,
                    const uint32_t* bits, const long long* tile_first, int64_t E, int64_t E_out,
                    int64_t* edges_out, unsigned char* shifts_out)
{
    chain_begin();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t mine = bits[(int64_t)blockIdx.x * 32 + lane];
    int total;
    const int before = warp_excl_scan(__popc(mine), lane, &total);
    const int64_t first = tile_first[blockIdx.x];
    // all edges of the thread are asked for before the first is written (one by one 51 us for 5.6 M edges, together 33)
    int64_t from[FILTER_ROUNDS], to[FILTER_ROUNDS], place[FILTER_ROUNDS];
    float h[FILTER_ROUNDS][3];
    const bool floats = shift_row_bytes == 12;
#pragma unroll
    for (int k = 0; k < FILTER_ROUNDS; k++) {
        const uint32_t word = __shfl_sync(0xffffffffu, mine, 8 * k + warp);
        const int64_t o = first + __shfl_sync(0xffffffffu, before, 8 * k + warp) + __popc(word & lanemask_lt());
        const int64_t e = (int64_t)blockIdx.x * FILTER_TILE + 256 * k + threadIdx.x;
        place[k] = ((word >> lane) & 1u) ? o : -1;
        if (place[k] < 0) continue;
        from[k] = edges[e];
        to[k] = edges[E + e];
        if (floats) {
            const float* a = reinterpret_cast<const float*>(shifts_raw) + 3 * e;
#pragma unroll
            for (int c = 0; c < 3; c++) h[k][c] = a[c];
        }
    }
#pragma unroll
    for (int k = 0; k < FILTER_ROUNDS; k++) {
        const int64_t o = place[k];
        if (o < 0) continue;
        edges_out[o] = from[k];
        edges_out[E_out + o] = to[k];
        if (floats) {
            float* b = reinterpret_cast<float*>(shifts_out) + 3 * o;
#pragma unroll
            for (int c = 0; c < 3; c++) b[c] = h[k][c];
        } else {
            const int64_t e = (int64_t)blockIdx.x * FILTER_TILE + 256 * k + threadIdx.x;
            for (int i = 0; i < shift_row_bytes; i++) shifts_out[o * shift_row_bytes + i] = shifts_raw[e * shift_row_bytes + i];
        }
    }
}

struct FilterLayout { int64_t tiles, bits, count, first, sums, total; };
static FilterLayout filter_layout(int64_t E)
{
    FilterLayout L;
    L.tiles = (E + FILTER_TILE - 1) / FILTER_TILE;
    int64_t o = 0;
    auto take = [&](int64_t bytes) { const int64_t r = o; o = align_up(o + bytes, 256); return r; };
    L.bits = take(L.tiles * 32 * 4);
    L.count = take(L.tiles * 4);
    L.first = take(L.tiles * 8);
    L.sums = take((int64_t)(scan_num_tiles(L.tiles) + 1) * 8);
    L.total = std::max<int64_t>(o, 256);
    return L;
}

static inline unsigned nblk(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace dynb

using namespace dynb;

// ------------------------------------------------------------------------------------------ C ABI
extern "C" int dynb_bincount_i64(const int64_t* a_dev, int64_t n, int64_t W, int64_t* counts_dev, uint32_t* bad_dev, void* stream)
{
    if (n < 0 || W < 1 || counts_dev == nullptr || bad_dev == nullptr) return fail_arg("bad arguments");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DYNB_CUDA_OK(clear_ranges(s, {counts_dev, W * 8, 0}, {bad_dev, 4, 0}));
    if (n == 0) return DYNB_OK;
    const int grid = (int)std::min<int64_t>(nblk(n), (int64_t)sm_count_cached() * 8);
    const size_t smem = W <= 4096 ? (size_t)W * 4 : 0;
    launch_chained(bincount_i64_kernel, grid, 256, smem, s, a_dev, n, W, reinterpret_cast<unsigned long long*>(counts_dev), bad_dev);
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

// workspace of a selection: matches per tile, then the sums of the prefix sum over them
static int64_t select_sums_at(int64_t n) { return align_up((n / SELECT_TILE + 1) * 4, 256); }

extern "C" int dynb_select_workspace_bytes(int64_t n, int64_t* bytes)
{
    if (n < 0 || bytes == nullptr) return fail_arg("bad arguments");
    // the edge filter takes a workspace of dynb_select_workspace_bytes(2 * E) too
    *bytes = std::max(select_sums_at(n) + align_up((int64_t)(scan_num_tiles(n / SELECT_TILE + 1) + 1) * 4, 256), filter_layout(n / 2).total);
    return DYNB_OK;
}

// out_dev must hold n elements (upper bound); *count_dev receives how many were written.
extern "C" int dynb_select_eq_i64(const int64_t* a_dev, int64_t n, int64_t value, const int64_t* gather_src_dev,
                                  int64_t* out_dev, int64_t* count_dev, void* workspace_dev, int64_t workspace_bytes,
                                  void* stream)
{
    if (n < 0 || count_dev == nullptr) return fail_arg("bad arguments");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n == 0) { DYNB_CUDA_OK(cudaMemsetAsync(count_dev, 0, 8, s)); return DYNB_OK; }
    int64_t need;
    dynb_select_workspace_bytes(n, &need);
    if (workspace_dev == nullptr || workspace_bytes < need) return fail_arg("workspace too small (see dynb_select_workspace_bytes)");
    uint32_t* tile_count = static_cast<uint32_t*>(workspace_dev);
    const unsigned tiles = nblk(n, SELECT_TILE);
    launch_chained(select_count_kernel, tiles, 256, 0, s, a_dev, n, value, tile_count);
    if (tiles <= SELECT_FUSED_MAX_TILES) {
        launch_chained(select_fill_kernel<false>, tiles, 256, 0, s, a_dev, n, value, tile_count, gather_src_dev, out_dev, count_dev);
    } else {
        uint32_t* sums = reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(workspace_dev) + select_sums_at(n));
        DYNB_CUDA_OK(cudaMemsetAsync(count_dev, 0, 8, s));
        DYNB_CUDA_OK((exclusive_scan<uint32_t, uint32_t>(tile_count, tile_count, nullptr, tiles, sums, reinterpret_cast<uint32_t*>(count_dev), s)));
        launch_chained(select_fill_kernel<true>, tiles, 256, 0, s, a_dev, n, value, tile_count, gather_src_dev, out_dev, count_dev);
    }
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

extern "C" int dynb_halo_mark_from_edges(const int64_t* edges_dev, int64_t E, const int64_t* pid_dev, int64_t N, int64_t my_rank,
                                         int64_t world_size, uint32_t* send_mask_dev, uint32_t* recv_mask_dev,
                                         uint8_t* has_remote_dev, uint32_t* bad_dev, void* stream)
{
    if (E < 0 || N < 0 || world_size < 1 || my_rank < 0 || my_rank >= world_size) return fail_arg("bad arguments");
    const int words = (int)((world_size + 31) / 32);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DYNB_CUDA_OK(clear_ranges(s, {send_mask_dev, N * words * 4, 0}, {recv_mask_dev, N * words * 4, 0}, {has_remote_dev, N, 0}, {bad_dev, 4, 0}));
    if (E == 0) return DYNB_OK;
    launch_chained(halo_mark_edges_kernel, nblk(E, MARK_EDGES * 256), 256, 0, s, edges_dev, edges_dev + E, E, pid_dev, N, my_rank, words, send_mask_dev,
                                                   recv_mask_dev, has_remote_dev, bad_dev);
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

static inline int hl_blocks(int64_t n) { return (int)std::max<int64_t>((n + HL_TILE - 1) / HL_TILE, 1); }

extern "C" int dynb_halo_lists_workspace_bytes(int64_t n, int64_t W, int64_t* bytes)
{
    if (n < 0 || W < 1 || bytes == nullptr) return fail_arg("bad arguments");
    *bytes = align_up((int64_t)hl_blocks(n) * (2 * W + 1) * 4, 256) + align_up((2 * W + 1) * 8, 256) + 256;
    return DYNB_OK;
}

static int halo_lists_args(const uint32_t* send_mask_dev, const uint32_t* recv_mask_dev, const int64_t* owner_dev, int64_t n, int64_t R,
                           int64_t W, HaloSets& h)
{
    if (n < 0 || W < 1) return fail_arg("bad arguments");
    if (n > 0 && (send_mask_dev == nullptr || (owner_dev == nullptr && recv_mask_dev == nullptr))) return fail_arg("null pointer");
    if (owner_dev != nullptr && (R < 0 || R >= W)) return fail_arg("rank out of range");
    if (W > 4096) return fail_arg("world_size above 4096 is not supported");
    h = HaloSets{send_mask_dev, recv_mask_dev, owner_dev, n, R, (int)((W + 31) / 32), (int)W};
    return DYNB_OK;
}

extern "C" int dynb_halo_lists_plan(const uint32_t* send_mask_dev, const uint32_t* recv_mask_dev, const int64_t* owner_dev, int64_t n,
                                    int64_t R, int64_t W, int64_t* offsets_dev, void* workspace_dev, int64_t workspace_bytes, void* stream)
{
    return dynb_halo_lists_plan_words(send_mask_dev, recv_mask_dev, owner_dev, n, R, W, offsets_dev, workspace_dev, workspace_bytes, nullptr, 0, stream);
}

extern "C" int dynb_halo_lists_plan_words(const uint32_t* send_mask_dev, const uint32_t* recv_mask_dev, const int64_t* owner_dev, int64_t n,
                                          int64_t R, int64_t W, int64_t* offsets_dev, void* workspace_dev, int64_t workspace_bytes,
                                          int64_t* words_host, int64_t n_words, void* stream)
{
    HaloSets h;
    int rc = halo_lists_args(send_mask_dev, recv_mask_dev, owner_dev, n, R, W, h);
    if (rc) return rc;
    int64_t need;
    dynb_halo_lists_workspace_bytes(n, W, &need);
    if (offsets_dev == nullptr) return fail_arg("null pointer");
    if (words_host != nullptr && (n_words < 0 || n_words > 2 * (W + 1) + 2)) return fail_arg("n_words out of range");
    if (workspace_dev == nullptr || workspace_bytes < need) return fail_arg("workspace too small (see dynb_halo_lists_workspace_bytes)");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int64_t* words_view = words_host != nullptr ? static_cast<int64_t*>(device_view_of_host(words_host)) : nullptr;
    if (n == 0) {
        DYNB_CUDA_OK(cudaMemsetAsync(offsets_dev, 0, (size_t)(2 * (W + 1) + 1) * 8, s));
        if (words_host != nullptr) DYNB_CUDA_OK(cudaMemcpyAsync(words_host, offsets_dev, (size_t)n_words * 8, cudaMemcpyDeviceToHost, s));
        return DYNB_OK;
    }
    const int nb = hl_blocks(n);
    unsigned char* ws = static_cast<unsigned char*>(workspace_dev);
    uint32_t* bsum = reinterpret_cast<uint32_t*>(ws);
    int64_t* totals = reinterpret_cast<int64_t*>(ws + align_up((int64_t)nb * (2 * W + 1) * 4, 256));
    uint32_t* arrived = reinterpret_cast<uint32_t*>(ws + need - 256);
    DYNB_CUDA_OK(clear_ranges(s, {arrived, 4, 0}));
    launch_chained(halo_lists_count_kernel, nb, HL_THREADS, 0, s, h, (int)W, nb, bsum);
    launch_chained(halo_lists_scan_kernel, (unsigned)(2 * W + 1), SCAN_THREADS, 0, s, bsum, nb, (int)W, totals, arrived, offsets_dev, words_view, (int)n_words);
    DYNB_CUDA_OK(cudaGetLastError());
    if (words_host != nullptr && words_view == nullptr)
        DYNB_CUDA_OK(cudaMemcpyAsync(words_host, offsets_dev, (size_t)n_words * 8, cudaMemcpyDeviceToHost, s));
    return DYNB_OK;
}

extern "C" int dynb_halo_lists_fill(const uint32_t* send_mask_dev, const uint32_t* recv_mask_dev, const int64_t* owner_dev, int64_t n,
                                    int64_t R, int64_t W, const int64_t* value_map_dev, const uint8_t* has_foreign_dev,
                                    const int64_t* offsets_dev, int64_t n_local, int64_t* send_local_dev, int64_t* recv_atom_dev,
                                    int64_t* recv_ghost_dev, uint8_t* interior_dev, int64_t* matrix_row_dev,
                                    const void* workspace_dev, void* stream)
{
    HaloSets h;
    int rc = halo_lists_args(send_mask_dev, recv_mask_dev, owner_dev, n, R, W, h);
    if (rc) return rc;
    if (n == 0) return DYNB_OK;
    if (offsets_dev == nullptr || workspace_dev == nullptr || (owner_dev == nullptr && value_map_dev == nullptr) ||
        (owner_dev != nullptr && has_foreign_dev == nullptr))
        return fail_arg("null pointer");
    const HaloListsOut out{value_map_dev, has_foreign_dev, send_local_dev, recv_atom_dev, recv_ghost_dev, interior_dev, matrix_row_dev, n_local};
    const int nb = hl_blocks(n);
    launch_chained(halo_lists_fill_kernel, nb, HL_THREADS, 0, static_cast<cudaStream_t>(stream), h, (int)W, nb, static_cast<const uint32_t*>(workspace_dev),
                                                                                   offsets_dev, out);
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

static inline int csr_blocks(int64_t n) { return (int)((n + CSR_THREADS - 1) / CSR_THREADS); }

extern "C" int dynb_csr_workspace_bytes(int64_t n, int64_t W, int64_t* bytes)
{
    if (n < 0 || W < 1 || bytes == nullptr) return fail_arg("bad arguments");
    *bytes = align_up((int64_t)std::max(csr_blocks(n), 1) * W * 4, 256) + align_up(W * 8, 256);
    return DYNB_OK;
}

extern "C" int dynb_csr_plan(const uint32_t* mask_dev, const int64_t* owner_dev, int64_t n, int64_t R, int mode, int64_t W,
                             int64_t* offsets_dev, void* workspace_dev, int64_t workspace_bytes, void* stream)
{
    if (n < 0 || W < 1 || mode < 0 || mode > 2 || offsets_dev == nullptr) return fail_arg("bad arguments");
    if (mode != CSR_RAW && owner_dev == nullptr) return fail_arg("owner required");
    if (W > 4096) return fail_arg("world_size above 4096 is not supported");
    int64_t need;
    dynb_csr_workspace_bytes(n, W, &need);
    if (workspace_dev == nullptr || workspace_bytes < need) return fail_arg("workspace too small (see dynb_csr_workspace_bytes)");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int words = (int)((W + 31) / 32);
    const int nb = std::max(csr_blocks(n), 1);
    unsigned char* ws = static_cast<unsigned char*>(workspace_dev);
    uint32_t* bsum = reinterpret_cast<uint32_t*>(ws);
    int64_t* totals = reinterpret_cast<int64_t*>(ws + align_up((int64_t)nb * W * 4, 256));
    if (n == 0) {
        DYNB_CUDA_OK(cudaMemsetAsync(offsets_dev, 0, (size_t)(W + 1) * 8, s));
        return DYNB_OK;
    }
    csr_count_kernel<<<nb, CSR_THREADS, 0, s>>>(mask_dev, words, owner_dev, n, R, mode, (int)W, nb, bsum);
    csr_scan_rows_kernel<<<(unsigned)W, SCAN_THREADS, 0, s>>>(bsum, nb, totals);
    csr_offsets_kernel<<<1, 32, 0, s>>>(totals, (int)W, offsets_dev);
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

extern "C" int dynb_csr_fill(const uint32_t* mask_dev, const int64_t* owner_dev, int64_t n, int64_t R, int mode, int64_t W,
                             const int64_t* value_map_dev, const int64_t* offsets_dev, int64_t* out_dev,
                             const void* workspace_dev, void* stream)
{
    if (n < 0 || W < 1 || mode < 0 || mode > 2) return fail_arg("bad arguments");
    if (n == 0) return DYNB_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int words = (int)((W + 31) / 32);
    const int nb = csr_blocks(n);
    const uint32_t* bsum = reinterpret_cast<const uint32_t*>(workspace_dev);
    csr_fill_kernel<<<nb, CSR_THREADS, 0, s>>>(mask_dev, words, owner_dev, n, R, mode, (int)W, nb, bsum, offsets_dev,
                                               value_map_dev, out_dev);
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

extern "C" int dynb_gather_not_u8(const uint8_t* flags_dev, const int64_t* idx_dev, int64_t n, uint8_t* out_dev, void* stream)
{
    if (n < 0) return fail_arg("bad arguments");
    if (n == 0) return DYNB_OK;
    launch_chained(gather_not_u8_kernel, nblk(n), 256, 0, static_cast<cudaStream_t>(stream), flags_dev, idx_dev, n, out_dev);
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

extern "C" int dynb_fill_bytes(void* at_dev, int64_t bytes, int byte, void* stream)
{
    if (bytes < 0 || (bytes > 0 && at_dev == nullptr)) return fail_arg("bad arguments");
    DYNB_CUDA_OK(clear_ranges(static_cast<cudaStream_t>(stream), {at_dev, bytes, (uint32_t)byte}));
    return DYNB_OK;
}

extern "C" int dynb_scatter_iota(const int64_t* idx_dev, int64_t n, int64_t N, int64_t* g2l_dev, uint32_t* bad_dev, void* stream)
{
    if (n < 0 || N < 0) return fail_arg("bad arguments");
    if (n == 0) return DYNB_OK;
    launch_chained(scatter_iota_kernel, nblk(n), 256, 0, static_cast<cudaStream_t>(stream), idx_dev, n, N, g2l_dev, bad_dev);
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

extern "C" int dynb_filter_edges_workspace_bytes(int64_t E, int64_t* bytes)
{
    if (E < 0 || bytes == nullptr) return fail_arg("bad arguments");
    *bytes = filter_layout(E).total;
    return DYNB_OK;
}

extern "C" int dynb_filter_edges_plan(const int64_t* edges_dev, const float* shifts_f32_dev, const float* pos_dev,
                                      const float* cell_host, double radius, int64_t E, int64_t* count_dev,
                                      void* workspace_dev, int64_t workspace_bytes, void* stream)
{
    if (E < 0 || count_dev == nullptr || cell_host == nullptr) return fail_arg("bad arguments");
    if (!(radius > 0.0)) return fail_arg("radius must be positive");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (E == 0) { DYNB_CUDA_OK(cudaMemsetAsync(count_dev, 0, 8, s)); return DYNB_OK; }
    const FilterLayout L = filter_layout(E);
    if (workspace_dev == nullptr || workspace_bytes < L.total) return fail_arg("workspace too small (see dynb_filter_edges_workspace_bytes)");
    unsigned char* ws = static_cast<unsigned char*>(workspace_dev);
    uint32_t* bits = reinterpret_cast<uint32_t*>(ws + L.bits);
    uint32_t* count = reinterpret_cast<uint32_t*>(ws + L.count);
    Cell9 c;
    for (int i = 0; i < 9; i++) c.c[i] = cell_host[i];
    const float r2 = static_cast<float>(radius * radius);  // dist_graph_ops_kernels.cu:84
    launch_chained(edge_keep_bits_kernel, (unsigned)L.tiles, 256, 0, s, edges_dev, edges_dev + E, shifts_f32_dev, pos_dev, c, r2, E, bits, count);
    DYNB_CUDA_OK((exclusive_scan<uint32_t, long long>(count, reinterpret_cast<long long*>(ws + L.first), nullptr, L.tiles,
                                                       reinterpret_cast<long long*>(ws + L.sums), reinterpret_cast<long long*>(count_dev), s)));
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

extern "C" int dynb_filter_edges_fill(const int64_t* edges_dev, const void* shifts_raw_dev, int shift_row_bytes, int64_t E,
                                      int64_t E_out, int64_t* edges_out_dev, void* shifts_out_dev, const void* workspace_dev,
                                      void* stream)
{
    if (E < 0 || E_out < 0 || shift_row_bytes <= 0) return fail_arg("bad arguments");
    if (E == 0 || E_out == 0) return DYNB_OK;
    const unsigned char* ws = static_cast<const unsigned char*>(workspace_dev);
    const FilterLayout L = filter_layout(E);
    launch_chained(edge_compact_kernel, (unsigned)L.tiles, 256, 0, static_cast<cudaStream_t>(stream), edges_dev, static_cast<const unsigned char*>(shifts_raw_dev), shift_row_bytes, reinterpret_cast<const uint32_t*>(ws + L.bits),
        reinterpret_cast<const long long*>(ws + L.first), E, E_out, edges_out_dev,
        static_cast<unsigned char*>(shifts_out_dev));
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}
