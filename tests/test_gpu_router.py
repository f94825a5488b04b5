"""Router projection (FP32 GEMM for batches, GEMV for a few rows, shared-router row fused) and the top-k margin audit, against
double-precision logits. The reference's forced-route fixture (native/tests/test_moe_mm_many_gpu.cpp:96-104) pins the ids."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tokspur_public_b200 import capi, synth  # noqa: E402
from tokspur_public_b200 import layer as L  # noqa: E402


def project(w, x, extra=None, x_pad=0, overflows=False):
    rows, cols = w.shape
    T = x.shape[0]
    dw = torch.from_numpy(w).cuda()
    xs = torch.full((T, cols + x_pad), -7654.25, dtype=torch.float32, device="cuda")
    xs[:, :cols] = torch.from_numpy(x).cuda()
    out = torch.full((T, rows + 4), -7654.25, dtype=torch.float32, device="cuda")
    de = torch.from_numpy(extra).cuda() if extra is not None else None
    eo = torch.zeros(T, dtype=torch.float32, device="cuda") if extra is not None else None
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    capi.call("tsp_router_project", dw.data_ptr(), rows, cols, de.data_ptr() if de is not None else None, xs.data_ptr(), (cols + x_pad) * 4, T,
              out.data_ptr(), (rows + 4) * 4, eo.data_ptr() if eo is not None else None, err.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert overflows or int(err.item()) == 0
    o = out.cpu().numpy()
    assert np.all(o[:, rows:] == np.float32(-7654.25))   # padding canaries untouched
    return o[:, :rows], (eo.cpu().numpy() if eo is not None else None)


@pytest.mark.parametrize("T", [1, 5, 40, 300, 1000])
@pytest.mark.parametrize("rows,cols", [(512, 2048), (130, 100)])
def test_router_projection_against_double(T, rows, cols):
    w = synth.normal(7 + rows, (rows, cols), 0.05)
    extra = synth.normal(9 + rows, (cols,), 0.05)
    x = synth.normal(11 + T, (T, cols))
    got, gex = project(w, x, extra, x_pad=4)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    wex = x.astype(np.float64) @ extra.astype(np.float64)
    scale = np.maximum(1.0, np.abs(want))
    assert np.max(np.abs(got - want) / scale) <= 5e-5
    assert np.max(np.abs(gex - wex) / np.maximum(1.0, np.abs(wex))) <= 5e-5


# Edges of the tensor-core product's tiles (128 token rows x 64 matrix rows x 64 columns, sums emptied every 256 columns), rows that are
# not whole 16-byte units, and the last batch of the one-warp-per-output form. Each value is the sum of three bfloat16 parts (8 + 8 + 8
# bits), the products left out are within 2^-24 of their term and a sum of n terms in FP32 keeps n * 2^-24 of its magnitude sum.
@pytest.mark.parametrize("T,rows,cols,pad", [(95, 65, 64, 0), (96, 1, 7, 0), (96, 64, 256, 4), (128, 63, 260, 0), (129, 130, 257, 3), (257, 65, 2048, 0)])
def test_router_projection_tile_edges(T, rows, cols, pad):
    w, x = synth.normal(3 + rows, (rows, cols), 0.05), synth.normal(5 + T, (T, cols))
    x[0] *= 1e30   # far outside binary16: the parts have FP32's range
    w[0] *= 1e-20
    got, _ = project(w, x, x_pad=pad)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    magnitude = np.abs(x.astype(np.float64)) @ np.abs(w.astype(np.float64)).T
    assert np.max(np.abs(got - want) / magnitude) <= (cols + 4) * 2.0 ** -24


# Few columns, where no other rounding hides what a split leaves out: significands whose parts are as large as they get (0x80ffff: parts cut
# off instead of rounded leave out 2^-21 of the product; 0x807fc0: the most that rounded parts leave out, 2^-24), random ones, and the
# largest finite value, which no bfloat16 rounds to. FP32: one rounding per term and the sum, here one more for what is left out.
@pytest.mark.parametrize("cols", [1, 2, 4])
def test_router_projection_keeps_every_bit_of_a_term(cols):
    rng = np.random.default_rng(cols)
    rows, T = 65, 130
    pick = lambda n: rng.choice(np.array([0x3f80ffff, 0x3f807fc0, 0xbf80ffff, 0x3f8000ff, 0x3fffffff], dtype=np.uint32), size=n).view(np.float32)
    w, x = pick((rows, cols)), pick((T, cols))
    w[32:], x[64:] = synth.normal(21, (rows - 32, cols)), synth.normal(22, (T - 64, cols))
    x[128:], w[0], w[40] = np.float32(3.4028235e38), 2.0 ** -20, 2.0 ** -30
    got, _ = project(w, x, overflows=True)   # the largest value times others than the two small rows
    x64, w64 = x.astype(np.float64), w.astype(np.float64)
    want, magnitude = x64 @ w64.T, np.abs(x64) @ np.abs(w64).T
    keep = magnitude < 3e38
    assert keep[128:].any()
    assert np.max((np.abs(got.astype(np.float64) - want) / magnitude)[keep]) <= (cols + 1.1) * 2.0 ** -24


# No further from 64-bit sums than an FP32 FMA chain over the columns (8.1e-7 at 2048, relative 2-norm); without the third part: 2.7e-6
@pytest.mark.parametrize("T,rows,cols", [(300, 512, 2048), (128, 64, 256), (96, 64, 64)])
def test_router_projection_is_as_exact_as_fp32(T, rows, cols):
    w, x = synth.normal(23, (rows, cols), 0.05), synth.normal(24, (T, cols))
    got, _ = project(w, x)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.linalg.norm(got - want) <= 8e-7 * np.linalg.norm(want)


def test_forced_route_fixture_ids_and_margins(oracle):
    E, Cn, K = 512, 64, 10
    w = np.zeros((E, Cn), np.float32)
    e = np.arange(E)
    w[:, 0] = (e - 8) / 32.0
    w[:, 1] = ((7 * e) % 17 - 8) / 16.0
    for T in (4, 130):   # the GEMV and the GEMM path
        x = np.zeros((T, Cn), np.float32)
        x[:, 0] = 1.0
        x[:, 1] = np.array([0.5, -0.5, 0.25, -0.25] * ((T + 3) // 4), np.float32)[:T]
        logits, _ = project(w, x)
        exact = x.astype(np.float64) @ w.astype(np.float64).T
        assert np.array_equal(logits.astype(np.float64), exact)   # every product and sum here is exact in binary32
        lg = torch.from_numpy(logits).cuda()
        ids = torch.zeros(T * K, dtype=torch.int32, device="cuda")
        wt = torch.zeros(T * K, dtype=torch.float32, device="cuda")
        mg = torch.zeros(T, dtype=torch.float32, device="cuda")
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        for mode in (0, 1):
            capi.call("tsp_moe_route_audit", lg.data_ptr(), E * 4, T, E, K, mode, 1, ids.data_ptr(), wt.data_ptr(), mg.data_ptr(), err.data_ptr(), L.stream_ptr())
            torch.cuda.synchronize()
            oi, ow = oracle.route_rows(exact, K, mode, True)
            assert np.array_equal(ids.cpu().numpy().view(np.uint32).reshape(T, K), oi)
            assert np.max(np.abs(wt.cpu().numpy().reshape(T, K) - ow)) <= 1e-6
            srt = np.sort(logits, axis=1)[:, ::-1]
            assert np.array_equal(mg.cpu().numpy(), (srt[:, K - 1] - srt[:, K]).astype(np.float32))
        assert int(err.item()) == 0
        tel = capi.RouterMarginTelemetry()
        fb = C.c_int(-1)
        capi.call("tsp_router_margin_evaluate", mg.data_ptr(), T, 1e-4, L.stream_ptr(), C.byref(tel), C.byref(fb))
        m = mg.cpu().numpy()
        assert tel.total_tokens == T and tel.total_layers == 1 and tel.violation_count == int((m <= 2e-4).sum())
        assert abs(tel.min_margin - float(m.min())) == 0 and abs(tel.sum_margin - float(m.astype(np.float64).sum())) <= 1e-9
        assert fb.value == int(tel.violation_count > 0) and tel.fallback_layers == fb.value


# Register form of the selection (up to 512 experts): few distinct values, both zeros, experts not a multiple of 32, every expert selected
@pytest.mark.parametrize("T,E,K", [(1, 512, 10), (9, 70, 64), (33, 512, 40), (64, 16, 16)])
def test_route_ties_and_signed_zeros(oracle, T, E, K):
    rng = np.random.default_rng(E + K)
    logits = rng.choice(np.array([-0.0, 0.0, 1.5, -2.25], dtype=np.float32), size=(T, E))
    lg = torch.from_numpy(logits).cuda()
    ids = torch.zeros(T * K, dtype=torch.int32, device="cuda")
    wt = torch.zeros(T * K, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for mode in (0, 1):
        capi.call("tsp_moe_route", lg.data_ptr(), E * 4, T, E, K, mode, 1, ids.data_ptr(), wt.data_ptr(), err.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        oi, ow = oracle.route_rows(logits.astype(np.float64), K, mode, True)
        assert np.array_equal(ids.cpu().numpy().view(np.uint32).reshape(T, K), oi)
        assert np.max(np.abs(wt.cpu().numpy().reshape(T, K) - ow)) <= 1e-6
    assert int(err.item()) == 0


# Infinities and NaN go through the three parts of the tensor-core product (130 rows) as through the FP32 chain (5): reported, and every other
# output as without them
@pytest.mark.parametrize("T", [5, 130])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_nonfinite_router_inputs(T, bad):
    rows, cols = 70, 256
    w, x = synth.normal(31, (rows, cols), 0.05), synth.normal(32, (T, cols))
    clean, _ = project(w, x)
    xb, wb = x.copy(), w.copy()
    xb[3, 9] = bad
    wb[66, 100] = bad
    for ww, xx, keep in ((w, xb, (np.arange(T) != 3)[:, None] & np.ones(rows, bool)), (wb, x, (np.arange(rows) != 66) & np.ones((T, 1), bool))):
        dw, dx = torch.from_numpy(ww).cuda(), torch.from_numpy(xx).cuda()
        out, err = torch.zeros((T, rows), dtype=torch.float32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        capi.call("tsp_router_project", dw.data_ptr(), rows, cols, None, dx.data_ptr(), cols * 4, T, out.data_ptr(), rows * 4, None, err.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert int(err.item()) & capi.ERR_NONFINITE
        assert np.array_equal(got[keep], clean[keep]) and not np.isfinite(got[~keep]).any()


def test_extra_row_of_the_largest_matrix_by_warps():
    """A warp per output: one row more than 2^27 outputs, numbered beyond what 32 bits of threads count."""
    rows, tokens = 1 << 21, 64
    w, x = torch.randn(rows, device="cuda"), torch.randn(tokens, device="cuda")
    extra = torch.tensor([1.5], device="cuda")
    out, extra_out, e = torch.full((tokens, rows), float("nan"), device="cuda"), torch.full((tokens,), float("nan"), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    capi.call("tsp_router_project", w.data_ptr(), rows, 1, extra.data_ptr(), x.data_ptr(), 4, tokens, out.data_ptr(), rows * 4, extra_out.data_ptr(), e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert int(e.item()) == 0
    assert torch.equal(extra_out, x * 1.5)
    for t in (0, 1, tokens - 1):
        assert torch.equal(out[t], w * x[t])
