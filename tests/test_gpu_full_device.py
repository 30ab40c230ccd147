"""An allocation that fails because the device is full: the call says so, and the next one, with
room again, is not failed by what the first left behind."""
import pytest
import torch

import scd_gb300
import scdgen

pytestmark = pytest.mark.gpu


def test_the_next_call_after_a_full_device():
    pairs = scdgen.rmat(19, 16, seed=1)   # about 0.8 GB while it is converted
    torch.zeros(1, device="cuda")
    with scd_gb300.Engine(0) as eng:
        eng.convert_edges(pairs[:2000])   # every kernel of it is loaded
        filler, left = [], torch.cuda.mem_get_info(0)[0] - (48 << 20)
        while left > 0:
            size = min(left, 1 << 36)
            filler.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            left -= size
        try:
            with pytest.raises(scd_gb300.ScdError) as ex:
                eng.convert_edges(pairs)
        finally:
            del filler
            torch.cuda.empty_cache()
        assert ex.value.status == -3
        eng.convert_edges(pairs)
        got = eng.graph_bytes()
    with scd_gb300.Engine(0) as eng:
        eng.convert_edges(pairs)
        assert eng.graph_bytes() == got
