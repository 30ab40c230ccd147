"""A conversion whose dense core has no room for its bit rows on a device that is nearly full:
counted by the walks instead, with the same bytes."""
import pytest
import torch

import scd_gb300
from test_gpu_core_widths import _ring

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    return torch.cuda.mem_get_info(0)[0]


def test_no_room_for_the_bit_rows():
    pairs = _ring(32768, False, 1)   # rows of 4 KB, two matrices: 256 MB
    torch.zeros(1, device="cuda")
    with scd_gb300.Engine(0, flags=scd_gb300.FLAG_TC_HASH) as eng:
        before = _free()
        eng.convert_edges(pairs)
        needed = before - _free()   # the device's pool keeps what the conversion used
        want = eng.graph_bytes()
    with scd_gb300.Engine(0, flags=scd_gb300.FLAG_PROFILE) as eng:
        eng.convert_edges(pairs[:2000])
        filler, left = [], _free() - needed - 100 * MB
        while left > 0:
            size = min(left, 1 << 36)
            filler.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            left -= size
        try:
            eng.convert_edges(pairs)
            cores = eng.profile("tc_dense")[1]
            got = eng.graph_bytes()
        finally:
            del filler
            torch.cuda.empty_cache()
        assert cores == 0 and got == want
        eng.convert_edges(pairs)   # with room again
        assert eng.profile("tc_dense")[1] == 1 and eng.graph_bytes() == want
