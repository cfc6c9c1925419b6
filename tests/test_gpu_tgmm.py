"""tgmm with 256-column tiles (two accumulators per CTA): the tile order, both ways to fetch the operands,
narrow last tiles and the choice between one CTA and a pair, against the oracle."""

import numpy as np
import pytest
import torch

from gpu_ragged_dot_b200 import _lib, ops
from oracle import ragged_dot_oracle as oracle
from tests import launched

pytestmark = pytest.mark.gpu
ONE, PAIR = "ragged_tgmm_kernel<1>", "ragged_tgmm_kernel<2>"
PLAIN = "ragged_gemm_kernel<256"  # tiles written one at a time


@pytest.mark.parametrize("dtype,rel", [(torch.bfloat16, 2e-3), (torch.float16, 3e-4)])
@pytest.mark.parametrize("m,k,n,g,kernel", [
    (40, 136, 264, 3, PLAIN),      # fewer tiles than CTAs
    (1300, 1000, 2384, 13, PAIR),  # two bands of column tiles, the last tile 80 wide, rows not of whole blocks
    (2275, 1016, 2176, 13, PAIR),  # the same with a last tile of 128 and whole blocks in n only
    (64, 504, 2176, 40, ONE),      # two rows per group
    (3200, 504, 2176, 40, PAIR),   # eighty
    (300, 392, 840, 60, ONE),      # output rows that split sectors, short groups
    (3000, 320, 2048, 3, PAIR),    # long groups: several stages per tile, one round
    (700, 1288, 776, 31, ONE),     # four tiles per row of 4, 3, 3 and 3 blocks, the order turned
    (500, 392, 1288, 30, ONE),     # six tiles, as many wide as narrow, turned
    (500, 392, 1392, 30, ONE),     # six tiles, rows of whole sectors, turned
    (500, 392, 2312, 20, ONE),     # ten tiles in two bands, turned
    (500, 392, 2320, 20, ONE),     # the same in whole sectors
    (500, 520, 1408, 30, ONE),     # rows of whole 256 bytes
    (700, 392, 1160, 17, PLAIN),   # five tiles, three rounds
    (700, 264, 1000, 40, PLAIN),   # four tiles, equally wide
    (300, 2048, 1160, 68, PLAIN),  # 37 rounds of tiles: loops run by one thread
    (500, 264, 136, 300, ONE),     # more groups than the table in shared memory holds; most rounds on one CTA
])
def test_tgmm_two_accumulators(m, k, n, g, kernel, dtype, rel):
    rng = np.random.default_rng(m + k)
    live = m - m // 10
    sizes = torch.from_numpy(rng.multinomial(live, rng.dirichlet(np.full(g, 0.7))).astype(np.int32))
    x = oracle.reference_normal(3 * m, (m, k), dtype)
    dout = oracle.reference_normal(3 * m + 1, (m, n), dtype)
    x[live:] = float("nan")  # rows of no group reach nothing
    dout[live:] = float("inf")
    want = oracle.trans_ragged_dot(x, dout, sizes).float()
    xd, dd, gd = x.cuda(), dout.cuda(), sizes.cuda()
    got, names = launched.kernels(lambda: ops.tgmm_forward(xd, dd, gd))
    assert any(kernel in name for name in names), names
    ws = ops._workspace(m, g, xd.device)
    for ctas in (1, 2):  # the same bits from either: the order of a contraction does not depend on the tile
        other = ops.tgmm_forward(xd, dd, gd, cfg=_lib.TileCfg(256, 0, ctas, 128), workspace=ws)
        assert ops.device_status(ws) == 0
        assert torch.equal(other, got)
    got = got.cpu().float()
    assert torch.isfinite(got).all()
    # float32 sums in another order, and one rounding to 16 bits (2^-9 or 2^-12 at most)
    assert float((got - want).norm() / want.norm()) < rel


@pytest.mark.parametrize("m,k,n,g,kernel", [
    (2570, 160, 4096, 10, "ragged_gemm_f32_pair_kernel"),  # three rounds of either; the peer's rows begin inside k
    (2570, 128, 4096, 10, "ragged_gemm_f32_kernel"),       # two rounds against three
    (2000, 160, 4096, 10, "ragged_gemm_f32_kernel"),       # groups of 200 and few rounds
    (1500, 1024, 4096, 10, "ragged_gemm_f32_pair_kernel"),  # of 150 in nine rounds
    (2570, 164, 4096, 10, "ragged_gemm_f32_kernel"),       # rows that are not multiples of 32
])
def test_float32_one_cta_or_pair(m, k, n, g, kernel):
    """Either side of the rule that puts one-pass float32 tgmm on pairs: the same TF32 products, added in the same
    order, so the bits of one CTA per tile; NaN in the rows of no group."""
    rng = np.random.default_rng(m + k)
    live = m - 70
    gs = torch.from_numpy(rng.multinomial(live, rng.dirichlet(np.full(g, 0.7))).astype(np.int32)).cuda()
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn((m, k), device="cuda", generator=gen)
    dout = torch.randn((m, n), device="cuda", generator=gen)
    x[live:], dout[live:] = float("nan"), float("nan")
    got, names = launched.kernels(lambda: ops.tgmm_forward(x, dout, gs))
    assert any(kernel in name for name in names), names
    one = ops.tgmm_forward(x, dout, gs, cfg=_lib.TileCfg(256, 0, 1, 128))
    assert torch.isfinite(got).all() and torch.equal(got, one)
