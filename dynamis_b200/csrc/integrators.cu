// Integrator steps for B200 (sm_100a), optionally fused with the drift word.
//
// Replaces the reference's integrator kernels (dynamis_integrator/src/csrc/euler_integrator.cu:9-26,
// verlet_integrator.cu:9-36, langevin_integrator.cu:9-52).  The per-component arithmetic is written with
// the same expression shapes, so that the compiler forms the same multiply-adds:
//   Euler        v += (f / m) * dt;               x += v * dt
//   Verlet 1     v += 0.5f * (f / m) * dt;        x += v * dt
//   Verlet 2     v += 0.5f * (f / m) * dt
//   Langevin 1   v = v * c1 + 0.5f * (f / m) * dt + c2 * noise;   x += v * dt
//   Langevin 2   v = (v + 0.5f * (f / m) * dt + c2 * noise) * c3
//   with c1 = 1 - 0.5 gamma dt, c2 = sqrt(gamma kT dt / m), c3 = 1 / (1 + 0.5 gamma dt).
// One thread owns whole atoms (three components), which lets the position-updating steps also produce the
// drift word of SimState.write_local_drift_flag (dynamis/src/dynamis/simulatorState.py:257-293) in the
// same pass over the state: the new positions and velocities are still in registers, so the watchdog
// costs the reference positions and the previous velocities (24 B/atom) instead of a second full pass.

#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace dynb {

enum { INT_EULER = 0, INT_VERLET1 = 1, INT_VERLET2 = 2, INT_LANGEVIN1 = 3, INT_LANGEVIN2 = 4 };

struct DriftArgs {
    const float* ref;     // [n,3] positions at the last rebuild
    float* prev_vel;      // [n,3] velocities of the previous step, overwritten
    uint32_t* state;      // 3 words, zero between calls
    int32_t* flag;        // the 2-bit word
    float threshold;
};

// One atom: its position x and velocity v are updated.
template <int KIND>
__device__ __forceinline__ void integrate_atom(float (&x)[3], float (&v)[3], const float (&f)[3], const float (&noise)[3], float m, float dt, float gamma, float kT)
{
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (KIND == INT_EULER) {
            v[k] += (f[k] / m) * dt;
        } else if (KIND == INT_VERLET1 || KIND == INT_VERLET2) {
            v[k] += 0.5f * (f[k] / m) * dt;
        } else if (KIND == INT_LANGEVIN1) {
            const float c1 = 1.0f - 0.5f * gamma * dt;
            const float c2 = sqrtf(gamma * kT * dt / m);
            v[k] = v[k] * c1 + 0.5f * (f[k] / m) * dt + c2 * noise[k];
        } else {
            const float c3 = 1.0f / (1.0f + 0.5f * gamma * dt);
            const float c2 = sqrtf(gamma * kT * dt / m);
            v[k] = (v[k] + 0.5f * (f[k] / m) * dt + c2 * noise[k]) * c3;
        }
        if (KIND == INT_EULER || KIND == INT_VERLET1 || KIND == INT_LANGEVIN1) x[k] += v[k] * dt;
    }
}
// Its distance from the reference and its reach within the next step (same expressions as drift_flag_kernel, state_ops.cu).
__device__ __forceinline__ void drift_atom(const float (&x)[3], const float (&v)[3], const float (&ref)[3], const float (&prev)[3], float dt, float& reach, float& disp)
{
    const float dx = x[0] - ref[0], dy = x[1] - ref[1], dz = x[2] - ref[2];
    const float vx = v[0], vy = v[1], vz = v[2];
    const float ax = vx - prev[0], ay = vy - prev[1], az = vz - prev[2];
    const float d = sqrtf(dx * dx + dy * dy + dz * dz);
    const float r = d + dt * (sqrtf(vx * vx + vy * vy + vz * vz) + sqrtf(ax * ax + ay * ay + az * az));
    disp = fmaxf(disp, d);
    reach = fmaxf(reach, r);
}

// A atoms a thread: with four of them an array's twelve numbers are three loads of 16 bytes (arrays that start on such a boundary; the
// up to three atoms behind the last four go one by one), else one atom and loads that lie 12 bytes apart.  Bound by HBM
// and, where the arrays stay in it, L2.  A Langevin step of 1 M atoms, both halves, drift word with the first, arrays out of L2: 42.2 us as
// two launches that wait for one another, 28.1 as a chain.
template <int KIND, bool DRIFT, int A>
__global__ void __launch_bounds__(256)
integrate_kernel(float* pos, float* vel, const float* frc, const float* mass, const float* noise, int64_t n, float dt, float gamma,
                 float kT, DriftArgs da)
{
    chain_begin();
    constexpr bool MOVES = KIND == INT_EULER || KIND == INT_VERLET1 || KIND == INT_LANGEVIN1, NOISE = KIND == INT_LANGEVIN1 || KIND == INT_LANGEVIN2;
    float reach = 0.0f, disp = 0.0f;
    auto load = [](const float* from, int64_t first, float (&to)[A][3]) {
        if constexpr (A == 4) {
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const float4 w = reinterpret_cast<const float4*>(from + 3 * first)[q];
                (&to[0][0])[4 * q] = w.x; (&to[0][0])[4 * q + 1] = w.y; (&to[0][0])[4 * q + 2] = w.z; (&to[0][0])[4 * q + 3] = w.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) to[0][k] = from[3 * first + k];
        }
    };
    auto store = [](float* to, int64_t first, const float (&from)[A][3]) {
        if constexpr (A == 4) {
#pragma unroll
            for (int q = 0; q < 3; q++)
                reinterpret_cast<float4*>(to + 3 * first)[q] = make_float4((&from[0][0])[4 * q], (&from[0][0])[4 * q + 1], (&from[0][0])[4 * q + 2], (&from[0][0])[4 * q + 3]);
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) to[3 * first + k] = from[0][k];
        }
    };
    const int64_t thread = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = thread; t < n / A; t += stride) {
        const int64_t i = A * t;
        float m[A], x[A][3] = {}, v[A][3], f[A][3], z[A][3] = {}, ref[A][3], prev[A][3];
        if constexpr (A == 4) {
            const float4 w = *reinterpret_cast<const float4*>(mass + i);
            m[0] = w.x; m[1] = w.y; m[2] = w.z; m[3] = w.w;
        } else {
            m[0] = mass[i];
        }
        load(vel, i, v);
        load(frc, i, f);
        if (NOISE) load(noise, i, z);
        if (MOVES) load(pos, i, x);
        if (DRIFT) {
            load(da.ref, i, ref);
            load(da.prev_vel, i, prev);
        }
#pragma unroll
        for (int a = 0; a < A; a++) {
            integrate_atom<KIND>(x[a], v[a], f[a], z[a], m[a], dt, gamma, kT);
            if (DRIFT) drift_atom(x[a], v[a], ref[a], prev[a], dt, reach, disp);
        }
        store(vel, i, v);
        if (MOVES) store(pos, i, x);
        if (DRIFT) store(da.prev_vel, i, v);
    }
    if (A > 1 && thread < n % A) {
        const int64_t i = n / A * A + thread;
        float x[3] = {0.0f, 0.0f, 0.0f}, v[3], f[3], z[3] = {0.0f, 0.0f, 0.0f}, ref[3], prev[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            v[k] = vel[3 * i + k];
            f[k] = frc[3 * i + k];
            if (NOISE) z[k] = noise[3 * i + k];
            if (MOVES) x[k] = pos[3 * i + k];
            if (DRIFT) { ref[k] = da.ref[3 * i + k]; prev[k] = da.prev_vel[3 * i + k]; }
        }
        integrate_atom<KIND>(x, v, f, z, mass[i], dt, gamma, kT);
        if (DRIFT) drift_atom(x, v, ref, prev, dt, reach, disp);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            vel[3 * i + k] = v[k];
            if (MOVES) pos[3 * i + k] = x[k];
            if (DRIFT) da.prev_vel[3 * i + k] = v[k];
        }
    }
    if (!DRIFT) return;
    // block maxima -> two atomics per block; the block that arrives last publishes the word and leaves
    // the state words zero for the next call (no block waits for another)
    __shared__ uint32_t sm[2][8];
    uint32_t rb = __float_as_uint(reach), db = __float_as_uint(disp);  // non-negative floats order like their bits
    rb = __reduce_max_sync(0xffffffffu, rb);
    db = __reduce_max_sync(0xffffffffu, db);
    if ((threadIdx.x & 31) == 0) { sm[0][threadIdx.x >> 5] = rb; sm[1][threadIdx.x >> 5] = db; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 0; w < 8; w++) { rb = max(rb, sm[0][w]); db = max(db, sm[1][w]); }
        atomicMax(&da.state[0], rb);
        atomicMax(&da.state[1], db);
        __threadfence();
        const uint32_t done = atomicAdd(&da.state[2], 1u);
        if (done == gridDim.x - 1) {
            __threadfence();
            const float R = __uint_as_float(atomicExch(&da.state[0], 0u));
            const float D = __uint_as_float(atomicExch(&da.state[1], 0u));
            da.state[2] = 0;
            *da.flag = ((R >= da.threshold) ? 1 : 0) + ((D > da.threshold) ? 2 : 0);
        }
    }
}

constexpr int64_t INT_L2_BYTES = 126ll << 20;

template <int KIND>
static int launch_integrator(float* pos, float* vel, const float* frc, const float* mass, const float* noise, int64_t n,
                             float dt, float gamma, float kT, const DriftArgs* da, cudaStream_t s)
{
    uintptr_t at = reinterpret_cast<uintptr_t>(pos) | reinterpret_cast<uintptr_t>(vel) | reinterpret_cast<uintptr_t>(frc) | reinterpret_cast<uintptr_t>(mass) |
                   reinterpret_cast<uintptr_t>(noise);
    if (da != nullptr) at |= reinterpret_cast<uintptr_t>(da->ref) | reinterpret_cast<uintptr_t>(da->prev_vel);
    // Four atoms a thread where the arrays outgrow L2, more threads with fewer loads each below.  One atom a thread and four, us a step with its arrays
    // in L2 / out of it: Langevin, both halves, drift word with the first (76 and 40 B an atom) 300 k atoms 14.8, 16.0 / 12.6, 12.5, 700 k
    // 20.3, 24.8 / 20.9, 22.5, 1 M 25.1, 30.9 / 28.1, 30.0, 2 M 56.2, 54.6 / 56.0, 53.7, 4 M 115.8, 111.2 / 113.2, 109.2; Euler (40 B)
    // 1 M 11.7, 14.1 / 12.4, 12.3, 2 M 17.7, 22.2 / 24.1, 21.9, 4 M 51.2, 47.9 / 47.8, 44.7.
    constexpr bool MOVES = KIND == INT_EULER || KIND == INT_VERLET1 || KIND == INT_LANGEVIN1, NOISE = KIND == INT_LANGEVIN1 || KIND == INT_LANGEVIN2;
    const int arrays = 2 + (MOVES ? 1 : 0) + (NOISE ? 1 : 0) + (da != nullptr ? 2 : 0);
    const bool wide = at % 16 == 0 && n * (12 * arrays + 4) >= INT_L2_BYTES;
    const int64_t threads = wide ? (n + 3) / 4 : n;
    const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((threads + 255) / 256, (int64_t)sm_count_cached() * 8));
    auto run = [&](auto drift, auto atoms) {
        return launch_chained(integrate_kernel<KIND, decltype(drift)::value, decltype(atoms)::value>, g, 256, 0, s, pos, vel, frc, mass, noise, n, dt, gamma, kT,
                              da != nullptr ? *da : DriftArgs{});
    };
    using one = std::integral_constant<int, 1>;
    using four = std::integral_constant<int, 4>;
    if (da != nullptr) DYNB_CUDA_OK(wide ? run(std::true_type(), four()) : run(std::true_type(), one()));
    else DYNB_CUDA_OK(wide ? run(std::false_type(), four()) : run(std::false_type(), one()));
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

}  // namespace dynb

using namespace dynb;

extern "C" int dynb_integrator_step(int kind, float* pos_dev, float* vel_dev, const float* frc_dev, const float* mass_dev,
                                    const float* noise_dev, int64_t n_atoms, double dt, double gamma, double kT,
                                    const float* drift_ref_dev, float* drift_prev_vel_dev, double drift_threshold,
                                    uint32_t* drift_state_dev, int32_t* drift_flag_dev, void* stream)
{
    if (kind < INT_EULER || kind > INT_LANGEVIN2) return fail_arg("kind must be 0 (Euler), 1/2 (Verlet half-steps) or 3/4 (Langevin half-steps)");
    if (n_atoms < 0) return fail_arg("n_atoms must be non-negative");
    const bool moves = (kind == INT_EULER || kind == INT_VERLET1 || kind == INT_LANGEVIN1);
    const bool langevin = (kind == INT_LANGEVIN1 || kind == INT_LANGEVIN2);
    const bool drift = drift_flag_dev != nullptr;
    if (drift && !moves) return fail_arg("the drift word can only ride on a step that moves the positions");
    if (drift && (drift_ref_dev == nullptr || drift_prev_vel_dev == nullptr || drift_state_dev == nullptr))
        return fail_arg("drift word requested: reference positions, previous velocities and state words are required");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n_atoms == 0) {
        if (drift) DYNB_CUDA_OK(cudaMemsetAsync(drift_flag_dev, 0, 4, s));
        return DYNB_OK;
    }
    if (vel_dev == nullptr || frc_dev == nullptr || mass_dev == nullptr || (moves && pos_dev == nullptr)) return fail_arg("null pointer");
    if (langevin && noise_dev == nullptr) return fail_arg("Langevin steps need a noise array");
    DriftArgs da{drift_ref_dev, drift_prev_vel_dev, drift_state_dev, drift_flag_dev, (float)drift_threshold};
    const DriftArgs* dp = drift ? &da : nullptr;
    const float fdt = (float)dt, fg = (float)gamma, fkT = (float)kT;
    switch (kind) {
        case INT_EULER: return launch_integrator<INT_EULER>(pos_dev, vel_dev, frc_dev, mass_dev, noise_dev, n_atoms, fdt, fg, fkT, dp, s);
        case INT_VERLET1: return launch_integrator<INT_VERLET1>(pos_dev, vel_dev, frc_dev, mass_dev, noise_dev, n_atoms, fdt, fg, fkT, dp, s);
        case INT_VERLET2: return launch_integrator<INT_VERLET2>(pos_dev, vel_dev, frc_dev, mass_dev, noise_dev, n_atoms, fdt, fg, fkT, dp, s);
        case INT_LANGEVIN1: return launch_integrator<INT_LANGEVIN1>(pos_dev, vel_dev, frc_dev, mass_dev, noise_dev, n_atoms, fdt, fg, fkT, dp, s);
        default: return launch_integrator<INT_LANGEVIN2>(pos_dev, vel_dev, frc_dev, mass_dev, noise_dev, n_atoms, fdt, fg, fkT, dp, s);
    }
}
