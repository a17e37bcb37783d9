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


def test_given_back_with_the_last_graph_and_by_trim():
    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    ctx.rmat(10, 1 << 12, 1).build().free()
    before = free_bytes()
    a = ctx.rmat(16, 1 << 25, 1).build()
    b = ctx.rmat(16, 1 << 24, 1).build()
    b.free()
    assert ctx.bytes_kept > 300 * MB
    held = ctx.bytes_in_use
    ctx.trim()
    assert ctx.bytes_kept == 0 and ctx.bytes_in_use <= held
    assert before - free_bytes() <= ctx.bytes_in_use + 64 * MB
    b = ctx.rmat(16, 1 << 24, 1).build()
    lv, _ = b.bfs(int(b.sample_roots(1, 1)[0]))
    assert lv.max() > 1
    b.free()
    a.free()
    assert ctx.bytes_kept == 0 and ctx.bytes_in_use == 0
    assert before - free_bytes() <= 64 * MB
    ctx.close()


def test_another_context_gets_the_kept_memory():
    """One context keeps 4 GB, torch holds all but 3 GB of the rest: another
    context's 5 GB graph fits, and torch's allocations are not in its way."""
    import torch

    import everythinggraph_gb300 as eg

    first, second = eg.Context(0), eg.Context(0)
    stays = first.er(1000, 1000, 1)
    first.er(1000, (4096 * MB) // 8, 1).free()
    assert first.bytes_kept >= 4096 * MB
    torch.cuda.empty_cache()
    fill = torch.empty(free_bytes() - 3072 * MB, dtype=torch.uint8, device="cuda")
    g = second.er(1000, (5120 * MB) // 8, 1)
    assert first.bytes_kept == 0
    g.free()  # little is free: not kept
    assert second.bytes_kept == 0
    del fill
    torch.cuda.empty_cache()
    stays.free()
    first.close()
    second.close()


def test_graphs_freed_by_another_thread():
    """A finaliser's thread frees graphs while the owner makes new ones."""
    import queue
    import threading

    import everythinggraph_gb300 as eg

    ctx = eg.Context(0)
    todo = queue.Queue()

    def free():
        while (g := todo.get()) is not None:
            g.free()

    t = threading.Thread(target=free)
    t.start()
    rng = np.random.default_rng(1)
    for m in rng.integers(1 << 14, 1 << 20, 400):
        todo.put(ctx.er(1000, int(m), 1))
    todo.put(None)
    t.join()
    assert ctx.bytes_in_use == 0 and ctx.bytes_kept == 0
    ctx.close()
