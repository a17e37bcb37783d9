"""Device memory that a context holds beyond its graphs' buffers: within the
budget, and given back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def free_bytes():
    import torch

    return torch.cuda.mem_get_info()[0]


def test_budget_caps_what_is_held():
    """Smaller buffers in the place of larger kept ones, up to the budget."""
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0, hbm_budget=4096 * MB)
    ctx.er(1000, 1000, 1).build(eg.CSR).free()
    before = free_bytes() + ctx.bytes_in_use

    def graphs(megabytes, count):
        return [ctx.er(1000, megabytes * MB // 8, 1) for _ in range(count)]

    for g in graphs(1000, 2):
        g.free()
    kept = graphs(890, 2) + graphs(2300, 1)
    assert before - free_bytes() <= (4096 + 16) * MB  # cudaMalloc's granularity
    with pytest.raises(eg.EGError) as e:
        graphs(300, 1)
    assert e.value.code == -3
    for g in kept:
        g.free()
    again = graphs(1000, 2)  # the same size is served from what is kept
    assert before - free_bytes() <= (4096 + 16) * MB
    del again
    ctx.close()
