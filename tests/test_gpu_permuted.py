"""GPU parity of the permutation-fused entry points (rd_gmm_permuted / rd_tgmm_permuted) through
the C ABI: against the CPU oracle, and bit-for-bit against the un-fused path (gather rows, then
rd_gmm / rd_tgmm on the sorted copy), which runs the same arithmetic in the same order."""

import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))

import gpu_ragged_dot_b200 as rd  # noqa: E402
from gpu_ragged_dot_b200 import _lib, ops  # noqa: E402
from oracle import ragged_dot_oracle as oracle  # noqa: E402
from tests import launched  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0) if torch.cuda.is_available() else None
RTOL = ATOL = 2e-2  # bf16 tolerance of the elementwise check


def _routing(seed, tokens, top_k, g, capacity_extra=0):
    """Top-k routing -> (group_sizes[g], in_rows[m], out_rows[m]) with m = tokens*top_k + extra.
    in_rows[r]: token feeding sorted row r; out_rows[r]: its slot token*top_k + j in the
    token-major expanded layout.  Entries past sum(group_sizes) are filled with junk."""
    rng = np.random.default_rng(seed)
    experts = np.stack([rng.permutation(g)[:top_k] for _ in range(tokens)])  # [tokens, top_k]
    flat = experts.reshape(-1)
    order = np.argsort(flat, kind="stable")
    gs = np.bincount(flat, minlength=g).astype(np.int32)
    in_rows = (order // top_k).astype(np.int32)
    out_rows = order.astype(np.int32)
    if capacity_extra:
        junk = rng.integers(-5, tokens + 5, size=capacity_extra).astype(np.int32)
        in_rows = np.concatenate([in_rows, junk])
        out_rows = np.concatenate([out_rows, junk])
    return torch.from_numpy(gs), torch.from_numpy(in_rows), torch.from_numpy(out_rows)


def _close(got, want, what):
    ok, worst = oracle.allclose_report(got, want, RTOL, ATOL)
    assert ok, f"{what}: worst violation {worst:.2f}x of |a-b| <= {ATOL} + {RTOL}|b|"


CASES = [
    # tokens, top_k, k, n, g, extra, tile_n
    (64, 2, 64, 64, 4, 0, None),
    (200, 2, 256, 384, 8, 0, None),
    (333, 4, 200, 328, 16, 37, None),
    (512, 1, 128, 256, 3, 0, 256),
    (300, 2, 192, 136, 8, 11, 128),
    (300, 2, 72, 72, 8, 0, 64),
]


@pytest.mark.parametrize("tokens,top_k,k,n,g,extra,tile_n", CASES)
@pytest.mark.parametrize("trans_rhs", [False, True])
def test_gmm_permuted(tokens, top_k, k, n, g, extra, tile_n, trans_rhs):
    gs, in_rows, out_rows = _routing(7, tokens, top_k, g, extra)
    m = in_rows.numel()
    total = int(gs.sum())
    x = oracle.reference_normal(11, (tokens, k), torch.bfloat16)
    A = oracle.reference_normal(12, (g, n, k) if trans_rhs else (g, k, n), torch.bfloat16)
    cfg = _lib.TileCfg(tile_n, 0, 0, 0, 0) if tile_n else None
    xd, Ad, gd, ird, ord_ = (t.to(DEV) for t in (x, A, gs, in_rows, out_rows))
    safe_in = in_rows.clamp(0, tokens - 1)

    # gather only: rows come back in sorted order, rows past sum(group_sizes) are zero
    ws = ops._workspace(m, g, DEV)
    y1 = ops.gmm_permuted_forward(xd, Ad, gd, in_rows=ird, trans_rhs=trans_rhs, cfg=cfg, workspace=ws)
    assert ops.device_status(ws) == 0
    want1 = oracle.ragged_dot(x[safe_in.long()], A, gs, trans_rhs=trans_rhs)
    _close(y1.cpu(), want1, "gather")
    if total < m:
        assert float(y1[total:].float().abs().max()) == 0.0
    unfused = ops.gmm_forward(ops.gather_rows(xd, ird.clamp(0, tokens - 1)), Ad, gd, trans_rhs=trans_rhs,
                              cfg=_lib.TileCfg(tile_n or 0, 0, 1, 128, 0))
    assert torch.equal(y1[:total], unfused[:total]), "fused gather differs from gather_rows + rd_gmm"

    # gather + scatter into the token-major expanded layout
    y_rows = tokens * top_k
    y2 = ops.gmm_permuted_forward(xd, Ad, gd, in_rows=ird, out_rows=ord_, y_rows=y_rows, trans_rhs=trans_rhs,
                                  cfg=cfg)
    want2 = oracle.ragged_dot_permuted(x, A, gs, in_rows=safe_in, out_rows=out_rows, y_rows=y_rows,
                                       trans_rhs=trans_rhs)
    _close(y2.cpu(), want2, "gather+scatter")
    inv = out_rows[:total].long().to(DEV)
    assert torch.equal(y2[inv], y1[:total]), "scattered rows differ from the sorted result"

    # scatter only, into a buffer that already holds data: untouched rows keep it
    xs = x[safe_in.long()].contiguous().to(DEV)
    base = torch.full((y_rows + 3, n), 7.0, dtype=torch.bfloat16, device=DEV)
    y3 = ops.gmm_permuted_forward(xs, Ad, gd, out_rows=ord_, out=base, m=m, trans_rhs=trans_rhs, cfg=cfg)
    assert y3.data_ptr() == base.data_ptr() or (n % 8)
    assert torch.equal(y3[inv], y1[:total])
    assert float((y3[y_rows:] - 7.0).float().abs().max()) == 0.0


@pytest.mark.parametrize("tokens,top_k,k,n,g,extra,tile_n", CASES)
def test_tgmm_permuted(tokens, top_k, k, n, g, extra, tile_n):
    gs, in_rows, out_rows = _routing(9, tokens, top_k, g, extra)
    m = in_rows.numel()
    x = oracle.reference_normal(21, (tokens, k), torch.bfloat16)
    dy = oracle.reference_normal(22, (tokens * top_k, n), torch.bfloat16)
    cfg = _lib.TileCfg(tile_n, 0, 0, 0, 0) if tile_n else None
    safe_in = in_rows.clamp(0, tokens - 1).long()
    safe_out = out_rows.clamp(0, tokens * top_k - 1).long()
    xs, dys = x[safe_in].contiguous(), dy[safe_out].contiguous()
    want = oracle.trans_ragged_dot(xs, dys, gs)
    xd, dyd, gd = x.to(DEV), dy.to(DEV), gs.to(DEV)
    ws = ops._workspace(m, g, DEV)
    got = ops.tgmm_permuted_forward(xd, dyd, gd, x_rows_index=in_rows.to(DEV), y_rows_index=out_rows.to(DEV),
                                    cfg=cfg, workspace=ws)
    assert ops.device_status(ws) == 0
    _close(got.cpu(), want, "tgmm both gathered")
    err = oracle.rel_l2_err(got.cpu(), want, axis=(-1, -2), mask=gs != 0)
    assert float(err.max()) < 2e-3
    for gi in (gs == 0).nonzero().flatten().tolist():
        assert float(got[gi].float().abs().max()) == 0.0
    unfused = ops.tgmm_forward(xs.to(DEV), dys.to(DEV), gd, cfg=_lib.TileCfg(tile_n or 0, 0, 1, 128, 0))
    assert torch.equal(got, unfused), "fused gathers differ from rd_tgmm on the sorted copies"
    # one side only
    got_x = ops.tgmm_permuted_forward(xd, dys.to(DEV), gd, x_rows_index=in_rows.to(DEV), m=m, cfg=cfg)
    assert torch.equal(got_x, unfused)
    got_y = ops.tgmm_permuted_forward(xs.to(DEV), dyd, gd, y_rows_index=out_rows.to(DEV), m=m, cfg=cfg)
    assert torch.equal(got_y, unfused)


@pytest.mark.parametrize("fused", [True, False, None])
def test_ragged_dot_permuted_vjp(fused):
    tokens, top_k, k, n, g = 150, 2, 96, 136, 6
    gs, in_rows, out_rows = _routing(3, tokens, top_k, g)
    x = oracle.reference_normal(31, (tokens, k), torch.bfloat16)
    A = oracle.reference_normal(32, (g, k, n), torch.bfloat16)
    dy = oracle.reference_normal(33, (tokens * top_k, n), torch.bfloat16)
    xd = x.to(DEV).requires_grad_(True)
    Ad = A.to(DEV).requires_grad_(True)
    y = rd.ops.ragged_dot_permuted(xd, Ad, gs.to(DEV), in_rows=in_rows.to(DEV), out_rows=out_rows.to(DEV),
                                   fused=fused)
    y.backward(dy.to(DEV))
    # oracle: the same composition, differentiated by hand with the reference's VJP wiring
    xs = x[in_rows.long()]
    dys = dy[out_rows.long()]
    dxs, dA = oracle.ragged_dot_vjp(xs, A, gs, dys)
    dx = torch.zeros((tokens, k), dtype=torch.float32).index_add_(0, in_rows.long(), dxs.float())
    _close(y.detach().cpu(), oracle.ragged_dot_permuted(x, A, gs, in_rows, out_rows, tokens * top_k), "fwd")
    _close(xd.grad.cpu(), dx.to(torch.bfloat16), "dx")
    _close(Ad.grad.cpu(), dA, "dA")


def test_permuted_argument_checks():
    lib = _lib.load()
    x = torch.zeros((16, 64), dtype=torch.bfloat16, device=DEV)
    A = torch.zeros((2, 64, 64), dtype=torch.bfloat16, device=DEV)
    gs = torch.tensor([8, 8], dtype=torch.int32, device=DEV)
    y = torch.zeros((16, 64), dtype=torch.bfloat16, device=DEV)
    ws = ops._workspace(16, 2, DEV)

    def call(**kw):
        a = dict(x_rows=16, in_rows=None, y_rows=16, out_rows=None, m=16, k=64, dtype=_lib.RD_DTYPE_BF16, cfg=None)
        a.update(kw)
        return lib.rd_gmm_permuted(x.data_ptr(), a["x_rows"], a["in_rows"], A.data_ptr(), 2, gs.data_ptr(), None,
                                   y.data_ptr(), a["y_rows"], a["out_rows"], ws.data_ptr(), ws.numel(), a["m"],
                                   a["k"], 64, 2, 0, a["dtype"], a["cfg"], None)

    assert call() == 0
    assert call(x_rows=8) == _lib.RD_ERR_BAD_SHAPE       # identity gather needs x_rows >= m
    assert call(y_rows=8) == _lib.RD_ERR_BAD_SHAPE       # identity scatter needs y_rows == m
    assert call(k=60) == _lib.RD_ERR_BAD_SHAPE
    assert call(dtype=_lib.RD_DTYPE_F32) == _lib.RD_ERR_BAD_DTYPE
    import ctypes
    pair = _lib.TileCfg(256, 0, 2, 0, 0)
    assert call(cfg=ctypes.byref(pair)) == _lib.RD_ERR_BAD_CONFIG
    torch.cuda.synchronize()


# ------------------------------------------------------------------ sum of rows by index, unwritten rows
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows_in,rows_out,cols,live", [
    (1, 1, 8, 1),
    (300, 7, 1032, 300),     # lists longer than a warp; 1032 = one 128-vector chunk and one vector
    (257, 400, 4096, 200),   # rows without a source; rows past the groups do not count
    (64, 64, 37, 64),        # rows that are not multiples of 16 bytes
    (500, 3, 64, 0),         # no live row
])
def test_sum_rows(dtype, rows_in, rows_out, cols, live):
    """Against a float64 sum: at most one rounding to the result's type (2^-9 bf16, 2^-12 fp16) plus
    float32 additions of up to 100 terms."""
    rng = np.random.default_rng(rows_in + cols)
    index = torch.from_numpy(rng.integers(-2, rows_out + 2, size=rows_in).astype(np.int32))
    src = oracle.reference_normal(3, (rows_in, cols), torch.float32).to(dtype)
    src[live:] = float("nan")
    gs = torch.tensor([live // 3, 0, live - live // 3], dtype=torch.int32)
    want = torch.zeros((rows_out, cols), dtype=torch.float64)
    mag = torch.zeros((rows_out, cols), dtype=torch.float64)
    idx = index[:live].long().clamp(0, rows_out - 1)
    want.index_add_(0, idx, src[:live].double())
    mag.index_add_(0, idx, src[:live].double().abs())
    got = ops.sum_rows(src.to(DEV), index.to(DEV), gs.to(DEV), rows_out)
    assert got.dtype == dtype
    again = ops.sum_rows(src.to(DEV), index.to(DEV), gs.to(DEV), rows_out)
    assert torch.equal(got, again)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 0.0}[dtype]
    bound = eps * want.abs() + (128 * 2.0 ** -24) * mag + 2.0 ** -24
    assert bool(((got.cpu().double() - want).abs() <= bound).all())


@pytest.mark.parametrize("rows_in,rows_out,live", [
    (32, 1, 32), (33, 1, 33),      # either side of what is ranked in registers
    (4096, 2, 4096),               # one window of indices
    (9001, 2, 9000),               # windows, the last one part full
    (9001, 150, 9001),             # lists of about 60 rows that span all windows
])
def test_sum_rows_adds_in_ascending_order(rows_in, rows_out, live):
    """Bit for bit the float32 sum in ascending order of the source rows, whatever the length of the lists:
    magnitudes over eight decades make any other order differ."""
    rng = np.random.default_rng(rows_in + rows_out)
    src = (rng.standard_normal((rows_in, 12)) * 10.0 ** rng.uniform(-4, 4, (rows_in, 1))).astype(np.float32)
    index = rng.integers(0, rows_out, size=rows_in).astype(np.int32)
    want = np.zeros((rows_out, 12), dtype=np.float32)
    for i in range(live):
        want[index[i]] += src[i]
    gs = torch.tensor([live], dtype=torch.int32, device=DEV)
    for _ in range(3):
        got = ops.sum_rows(torch.from_numpy(src).to(DEV), torch.from_numpy(index).to(DEV), gs, rows_out)
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("tokens,extra,y_rows", [(96, 0, 192), (96, 33, 200), (5, 0, 300), (96, 33, 190000)])
def test_gmm_permuted_clears_unnamed_rows(tokens, extra, y_rows):
    """Rows of y that no sorted row names are zero, also where memory held something else."""
    g, k, n = 4, 64, 136
    gs, in_rows, out_rows = _routing(11, tokens, 2, g, extra)
    out_rows = torch.where(out_rows % 7 == 0, out_rows + 1000, out_rows)  # some destinations do not exist
    x = oracle.reference_normal(1, (tokens, k), torch.bfloat16)
    A = oracle.reference_normal(2, (g, k, n), torch.bfloat16)
    junk = torch.full((y_rows, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    del junk  # the allocator hands this block out again
    y = ops.gmm_permuted_forward(x.to(DEV), A.to(DEV), gs.to(DEV), in_rows=in_rows.to(DEV), out_rows=out_rows.to(DEV),
                                 y_rows=y_rows).cpu()
    named = torch.zeros(y_rows, dtype=torch.bool)
    live = out_rows[: int(gs.sum())].long()
    named[live[(live >= 0) & (live < y_rows)]] = True
    assert torch.equal(y[~named], torch.zeros_like(y[~named]))
    assert torch.isfinite(y.float()).all() and bool((y[named].abs().sum(1) > 0).all())


@pytest.mark.parametrize("y_rows,marks", [(1 << 14, False), (3 << 15, True)])
def test_small_results_are_cleared_whole(y_rows, marks):
    """Rows of 512 bytes: 8 MB of result are cleared by one memset, 48 MB by marking what is written."""
    g, k, n = 2, 64, 256
    gs, in_rows, out_rows = _routing(3, 64, 1, g)
    x = oracle.reference_normal(1, (64, k), torch.bfloat16).to(DEV)
    A = oracle.reference_normal(2, (g, k, n), torch.bfloat16).to(DEV)
    args = [t.to(DEV) for t in (gs, in_rows, out_rows)]
    y, names = launched.kernels(lambda: ops.gmm_permuted_forward(x, A, args[0], in_rows=args[1], out_rows=args[2],
                                                                   y_rows=y_rows))
    assert any("mark_rows" in name for name in names) == marks
    rows = torch.zeros(y_rows, dtype=torch.bool)
    rows[out_rows.long()] = True
    assert bool((y.cpu().float().abs().sum(1) > 0).eq(rows).all())


@pytest.mark.parametrize("trans_rhs", [False, True])
def test_long_groups_gather_and_scatter_in_one_kernel(trans_rhs):
    """The route a call with long groups takes: one product that gathers and scatters itself, nothing gathered
    before it; bit-equal to gather_rows, the plain product and a scatter, junk indices past the
    groups and destinations that do not exist included."""
    tokens, g, k, n = 4400, 2, 136, 2048 * 8
    gs, in_rows, out_rows = _routing(5, tokens, 1, g, 77)
    out_rows = torch.where(out_rows % 11 == 0, out_rows - 100000, out_rows)
    in_rows[3] = tokens + 9  # a zero row
    x = oracle.reference_normal(1, (tokens, k), torch.bfloat16).to(DEV)
    A = oracle.reference_normal(2, (g, n, k) if trans_rhs else (g, k, n), torch.bfloat16).to(DEV)
    gd, ird, ord_ = gs.to(DEV), in_rows.to(DEV), out_rows.to(DEV)
    ys = ops.gmm_forward(ops.gather_rows(x, ird), A, gd, trans_rhs=trans_rhs)
    live = torch.arange(ird.numel(), device=DEV) < int(gs.sum())
    named = live & (ord_ >= 0) & (ord_ < tokens)
    want = torch.zeros((tokens, n), dtype=torch.bfloat16, device=DEV)
    want[ord_[named].long()] = ys[named]
    got, names = launched.kernels(lambda: rd.ragged_dot_permuted(x, A, gd, in_rows=ird, out_rows=ord_, y_rows=tokens,
                                                         trans_rhs=trans_rhs))
    assert torch.equal(got, want)
    assert sum("ragged_gemm" in name for name in names) == 1 and any("ragged_gemm_perm" in name for name in names)
    assert not any("gather_rows" in name for name in names)
