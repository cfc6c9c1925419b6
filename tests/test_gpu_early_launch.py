"""Kernels that start before the kernel in front of them has finished: which calls do, read from the edges of a
captured graph, and that what they compute does not depend on it."""

import ctypes

import pytest
import torch

from gpu_ragged_dot_b200 import ops
from tests import launched

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _capture(fn):
    """fn captured: the graph, what fn returned, and for every edge whether it lets its end start early."""
    graph, res = launched.graph_of(fn)
    get = ctypes.CDLL("libcudart.so.12").cudaGraphGetEdges_v2
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert get(handle, None, None, None, ctypes.byref(n)) == 0
    starts, stops, data = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (ctypes.c_uint8 * (8 * n.value))()
    assert get(handle, starts, stops, data, ctypes.byref(n)) == 0
    return graph, res, [data[8 * i + 2] == 1 for i in range(n.value)]  # byte 2: the type, 1 = programmatic


@pytest.mark.parametrize("op,m,k,n,g,dtype,early", [
    ("gmm", 4096, 264, 256, 64, torch.bfloat16, True),      # one tile per CTA at most
    ("gmm", 4096, 264, 1024, 64, torch.bfloat16, True),     # 64 rows per group
    ("gmm", 4097, 264, 1024, 64, torch.bfloat16, False),    # a row more
    ("gmm", 640, 2000, 2000, 64, torch.bfloat16, True),     # 256 million weights
    ("gmm", 640, 2000, 2008, 64, torch.bfloat16, False),
    ("gmm", 640, 2000, 2000, 64, torch.float32, True),      # counted, not measured in bytes
    ("gmm", 640, 2000, 2004, 64, torch.float32, False),
    ("gmm_t", 640, 1024, 1144, 64, torch.bfloat16, True),   # 75 million with rows along the contraction
    ("gmm_t", 640, 1024, 1152, 64, torch.bfloat16, False),
    ("gmm_t", 640, 1024, 1152, 64, torch.float32, False),
    ("gmm3_t", 640, 1024, 1152, 64, torch.float32, True),   # three products: on CTA pairs, the larger limit
    ("tgmm", 640, 2000, 2000, 64, torch.bfloat16, True),
    ("tgmm", 640, 2000, 2008, 64, torch.bfloat16, False),
    ("tgmm", 16, 2000, 2008, 64, torch.float32, True),      # 16 groups at most have rows
    ("tgmm", 1000, 520, 1024, 14, torch.bfloat16, True),    # two tiles per CTA at most (280 tiles)
    ("tgmm", 1000, 520, 1024, 15, torch.bfloat16, False),   # 300
    ("tgmm", 2000, 520, 1024, 2, torch.bfloat16, True),     # 24 on pairs
    ("tgmm", 1000, 520, 1024, 14, torch.float32, False),    # float32: one tile per CTA
])
def test_which_calls_start_early(op, m, k, n, g, dtype, early):
    gs = torch.full((g,), m // g, dtype=torch.int32, device=DEV)
    x = torch.ones((m, k), dtype=dtype, device=DEV)
    if op == "tgmm":
        y = torch.ones((m, n), dtype=dtype, device=DEV)
        call = lambda: ops.tgmm_forward(x, y, gs)  # noqa: E731
    else:
        trans = op.endswith("_t")
        A = torch.ones((g, n, k) if trans else (g, k, n), dtype=dtype, device=DEV)
        cfg = ops._THREE_PASS if op == "gmm3_t" else None
        call = lambda: ops.gmm_forward(x, A, gs, trans_rhs=trans, cfg=cfg)  # noqa: E731
    graph, _, edges = _capture(lambda: (call(), call()))
    assert edges == [early]
    graph.reset()


@pytest.mark.parametrize("dtype,cfg", [(torch.bfloat16, None), (torch.float32, None), (torch.float32, ops._THREE_PASS)])
def test_short_groups_in_a_row(dtype, cfg):
    """Short groups with several tiles per CTA, each product reading what the one before it wrote, and results let go
    of as they are used up, so that later ones are written where earlier ones were still being read: the bits of the
    same calls with a synchronisation between them, in a stream and replayed as a graph on new inputs."""
    m, k, n, g = 2000, 512, 1024, 64
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((m, k), device=DEV, generator=gen).to(dtype)
    A = (torch.randn((g, k, n), device=DEV, generator=gen) / k ** 0.5).to(dtype)
    sizes = torch.randint(0, 54, (g,), generator=torch.Generator().manual_seed(6))
    sizes[3], sizes[40] = 0, 131
    assert m - 200 < int(sizes.sum()) <= m
    gs = sizes.to(torch.int32).to(DEV)

    def chain(sync):
        def step(fn, *args, **kw):
            res = fn(*args, cfg=cfg, **kw)
            if sync:
                torch.cuda.synchronize()
            return res

        kept = []
        for _ in range(3):
            y = step(ops.gmm_forward, x, A, gs)
            dx = step(ops.gmm_forward, y, A, gs, trans_rhs=True)
            dA = step(ops.tgmm_forward, dx, y, gs)
            del y
            z = step(ops.gmm_forward, dx, dA, gs)
            del dx
            kept.append(step(ops.gmm_forward, z, dA, gs, trans_rhs=True))
        return kept

    want = chain(True)
    for _ in range(3):
        for a, b in zip(chain(False), want):
            assert torch.equal(a, b)
    graph, got, edges = _capture(lambda: chain(False))
    assert edges == [True] * 14  # fifteen launches, every one allowed to start early
    scale = 2.0
    x.mul_(scale)  # exact: x enters the results five times
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b * scale ** 5)
    graph.reset()
