"""gmm with rows on the N side: rows dealt to tiles in steps of 16, and groups visited by the height of their
tiles, against 128-row tiles that multiply the same operands in the order of the groups."""

import numpy as np
import pytest
import torch

from gpu_ragged_dot_b200 import _lib, ops
from tests import launched

pytestmark = pytest.mark.gpu
# around whole steps, tiles and both: 1 row, 16 and 32 more or less one, one tile and a row, 17 blocks for two tiles
EDGES = [1, 15, 16, 17, 31, 32, 33, 47, 0, 255, 256, 257, 272, 273, 511, 512, 513, 528, 0, 1500, 3000]


@pytest.mark.parametrize("m,k,n,g,over", [
    (11000, 576, 8192, 21, 0),     # every edge, heights in no order
    (11000, 600, 8184, 21, 700),   # sizes that add up to more rows than there are: the last group is cut
    (131072, 576, 512, 256, 0),    # as many groups as the table in shared memory holds
])
def test_rows_in_steps_of_16(m, k, n, g, over):
    rng = np.random.default_rng(m + g)
    sizes = np.array((EDGES * (g // len(EDGES) + 1))[:g])
    rng.shuffle(sizes)
    sizes[int(rng.integers(g))] += m + over - 5 - sizes.sum()  # the last five rows in no group
    gs = torch.from_numpy(sizes.astype(np.int32)).cuda()
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn((m, k), device="cuda", generator=gen).bfloat16()
    w = torch.randn((g, n, k), device="cuda", generator=gen).bfloat16()
    if not over:
        x[m - 5:] = float("nan")
    whole = _lib.TileCfg(256, 0, 1, 128, 0)
    ws = ops._workspace(m, g, x.device)
    for weights, trans in ((w, True), (w.transpose(1, 2).contiguous(), False)):
        if not trans and n % 64:
            continue
        got, names = launched.kernels(lambda: ops.gmm_forward(x, weights, gs, trans_rhs=trans, workspace=ws,
                                                              cfg=_lib.TileCfg(0, 0, 0, 0, 0)))
        assert any("ragged_gemm_swap_kernel" in name for name in names), names
        assert ops.device_status(ws) == 0
        ref = ops.gmm_forward(x, weights, gs, trans_rhs=trans, cfg=whole).float()
        # the same products summed in fp32: a result differs by one rounding to 16 bits at most
        assert torch.isfinite(got).all()
        assert float(((got.float() - ref).abs() - 2.0 ** -7 * ref.abs()).max()) <= 1e-4 * float(ref.abs().max())
        if not over:
            assert float(got[m - 5:].abs().max()) == 0.0


@pytest.mark.parametrize("m,k,n,g,trans", [
    (11000, 388, 4096, 21, False),   # the fewest rounds it takes, every edge of a tile's rows; k ends inside a stage
    (11000, 388, 4092, 21, True),    # n ends inside a block of 32 columns
    (5001, 1032, 6176, 3, False),    # n ends a block of 32 into a tile
])
def test_float32_rows_in_steps_of_16(m, k, n, g, trans):
    rng = np.random.default_rng(m + n)
    sizes = np.array(EDGES if g == len(EDGES) else [1000, 0, 1500])
    rng.shuffle(sizes)
    sizes[int(rng.integers(g))] += m - 5 - sizes.sum()
    gs = torch.from_numpy(sizes.astype(np.int32)).cuda()
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn((m, k), device="cuda", generator=gen)
    w = torch.randn((g, n, k) if trans else (g, k, n), device="cuda", generator=gen)
    x[m - 5:] = float("nan")
    ws = ops._workspace(m, g, x.device)
    got, names = launched.kernels(lambda: ops.gmm_forward(x, w, gs, trans_rhs=trans, workspace=ws,
                                                          cfg=_lib.TileCfg(0, 0, 0, 0, 0)))
    assert any("ragged_gemm_swap_kernel" in name for name in names), names
    assert ops.device_status(ws) == 0
    ref = ops.gmm_forward(x, w, gs, trans_rhs=trans, cfg=_lib.TileCfg(256, 0, 1, 128, 0))
    assert torch.equal(got[:m - 5], ref[:m - 5])  # the same TF32 products, added in the same order
    assert float(got[m - 5:].abs().max()) == 0.0


@pytest.mark.parametrize("dtype,m,k,n,swapped", [
    (torch.float32, 590, 8192, 12640, False),        # 75 tiles for 74 pairs
    (torch.float32, 512, 8192, 12640, True),         # 50, in one round against two
    (torch.float8_e4m3fn, 338, 8416, 12520, False),  # one round of either kernel
    (torch.bfloat16, 1785, 4096, 4672, True),        # 70 tiles
])
def test_one_group_is_counted(dtype, m, k, n, swapped):
    """The rule for few rounds on one group, whose tiles the host can count."""
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn((m, k), device="cuda", generator=gen).to(dtype)
    w = torch.randn((1, n, k), device="cuda", generator=gen, dtype=torch.bfloat16).to(dtype)
    gs = torch.tensor([m - 3], dtype=torch.int32, device="cuda")
    fn = ops.gmm_fp8_forward if dtype == torch.float8_e4m3fn else lambda *a, **kw: ops.gmm_forward(*a, trans_rhs=True, **kw)
    got, names = launched.kernels(lambda: fn(x, w, gs))
    assert any("ragged_gemm_swap_kernel" in name for name in names) == swapped, names
    ref = fn(x, w, gs, cfg=_lib.TileCfg(256, 0, 1, 128, 0))
    assert float((got.float() - ref.float()).abs().max()) <= 2.0 ** -7 * float(ref.float().abs().max())
    assert float(got[m - 3:].float().abs().max()) == 0.0
