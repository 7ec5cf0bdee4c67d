"""The number of values up to which a selection writes its count without a prefix sum over its tiles is stated twice."""

import pathlib
import re

from dynamis_b200 import partition


def test_limit_is_the_kernels():
    source = (pathlib.Path(partition.__file__).parent / "csrc" / "halo.cu").read_text()
    value = {name: int(re.search(rf"constexpr \w+ {name} = (\d+);", source).group(1)) for name in ("SELECT_TILE", "SELECT_FUSED_MAX_TILES")}
    assert partition.SELECT_HOST_COUNT == value["SELECT_TILE"] * value["SELECT_FUSED_MAX_TILES"]
