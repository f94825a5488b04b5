"""The five-bit encodings of the reference's model on the decode-size path: Q5_K gate / up tensors and Q5_1 down tensors
(model.cpp:50-57; decoders numeric.cpp:38-50), plain GGUF rows. Dequantised weights bit-exact against the CPU oracle (which is
pinned to the reference's decoder and its fixture blocks); projections and whole layers within the reference's 5e-5 scaled
error (ffn_check.cpp:48-55)."""
import ctypes as C

import numpy as np
import pytest

import fixtures

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tokspur_public_b200 import capi, formats, synth  # noqa: E402
from tokspur_public_b200 import layer as L  # noqa: E402

DEV = "cuda"


def scaled_error(actual, expected):
    return float(np.max(np.abs(actual.astype(np.float64) - expected) / np.maximum(1.0, np.abs(expected))))


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


@pytest.mark.parametrize("type_", [formats.Q5_K, formats.Q5_1])
def test_dequant_bit_exact(oracle, type_):
    cols, rows, E = 512, 16, 2
    for w in (fixtures.lcg_weights(type_, cols, rows, E),      # every bit pattern of codes and factors, extreme scales
              np.stack([formats.quantize(type_, synth.normal(40 + e, (rows, cols), 0.02)).reshape(-1) for e in range(E)])):
        t = dev(w)
        ms = L.matrix_set(t, type_, formats.GGUF, rows, cols, E)
        out = torch.empty(rows * cols, dtype=torch.float32, device=DEV)
        e = torch.zeros(1, dtype=torch.int32, device=DEV)
        for ex in range(E):
            capi.call("tsp_dequant_f32", C.byref(ms), ex, out.data_ptr(), e.data_ptr(), L.stream_ptr())
            got = out.cpu().numpy()
            assert np.array_equal(got.view(np.uint32), oracle.dequantize(type_, w[ex], rows * cols).view(np.uint32))
        torch.cuda.synchronize()
        assert int(e.item()) == 0


def test_planar_layout_is_refused():
    t = torch.zeros(16 * 2 * 176, dtype=torch.uint8, device=DEV)
    ms = L.matrix_set(t, formats.Q5_K, formats.GGUF, 16, 512, 1)
    ms.layout = formats.PLANAR
    out = torch.empty(16 * 512, dtype=torch.float32, device=DEV)
    e = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert capi.lib().tsp_dequant_f32(C.byref(ms), 0, out.data_ptr(), e.data_ptr(), L.stream_ptr()) != 0
    assert capi.lib().tsp_expert_bytes(formats.Q5_K, formats.PLANAR, 16, 512) == 0


@pytest.mark.parametrize("type_,rows,cols,T", [(formats.Q5_K, 64, 512, 5), (formats.Q5_1, 96, 256, 16), (formats.Q5_K, 32, 2048, 11), (formats.Q5_1, 16, 64, 1)])
def test_dense_projection_against_oracle(oracle, type_, rows, cols, T):
    w = formats.quantize(type_, synth.normal(51, (rows, cols), 0.02)).reshape(-1)
    t = dev(w)
    ms = L.matrix_set(t, type_, formats.GGUF, rows, cols, 1)
    x = synth.normal(52, (T, cols), 1.0)
    dx = dev(x)
    out = torch.zeros((T, rows), dtype=torch.float32, device=DEV)
    e = torch.zeros(1, dtype=torch.int32, device=DEV)
    capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, 1, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert int(e.item()) == 0
    want = np.stack([oracle.gemv(type_, w, cols, rows, x[i]) for i in range(T)])
    assert scaled_error(out.cpu().numpy(), want) <= 5e-5


# The MMA kernel's edges: one warp's rows, a block's and more; tiles of up to four rows (low halves in the free columns) and of more; the
# shortest K; activations far outside binary16's range. A value keeps 22 bits (high + low half) and an FP32 sum of n terms n * 2^-24 of its
# magnitude sum, a term being the activation times the scaled code or the offset, each at most twice the largest weight; a tile's size
# may not show in a row's result.
@pytest.mark.parametrize("type_,rows,cols", [(formats.Q5_K, 16, 256), (formats.Q5_K, 144, 2048), (formats.Q5_1, 16, 128), (formats.Q5_1, 272, 512)])
def test_dense_projection_tile_edges(oracle, type_, rows, cols):
    w = formats.quantize(type_, synth.normal(81, (rows, cols), 0.02)).reshape(-1)
    t = dev(w)
    ms = L.matrix_set(t, type_, formats.GGUF, rows, cols, 1)
    x = synth.normal(82, (8, cols), 1.0)
    x[1] *= 1e30
    x[2] *= 1e-25
    x[3] = 0.0
    x[4, 0] = 65000.0
    w64 = oracle.dequantize(type_, w, rows * cols).astype(np.float64).reshape(rows, cols)
    want = x.astype(np.float64) @ w64.T
    magnitude = 4 * np.abs(w64).max() * np.abs(x.astype(np.float64)).sum(axis=1)[:, None]
    dx, alone = dev(x), []
    e = torch.zeros(1, dtype=torch.int32, device=DEV)
    for T in (8, 5, 4, 1):
        out = torch.zeros((T, rows), dtype=torch.float32, device=DEV)
        capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, 1, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert np.all(np.abs(got - want[:T]) <= (cols + 8) * 2.0 ** -24 * magnitude[:T])
        alone.append(got)
    assert int(e.item()) == 0
    for a in alone[1:]:
        assert np.array_equal(a, alone[0][:len(a)])


# Both kernels on the same eight rows (a batch of sixteen takes the FP32 FMA kernel): the split into binary16 halves and the sums of the MMA
# kernel may not be further from 64-bit sums than the FP32 kernel's are. (Summed in one chain over K instead of step by step: 2.2e-7
# against 1.6e-7 at 2048 columns. High halves alone: 2e-4.)
@pytest.mark.parametrize("type_,rows,cols", [(formats.Q5_K, 256, 2048), (formats.Q5_K, 256, 256), (formats.Q5_1, 512, 512), (formats.Q5_1, 256, 2048), (formats.Q5_1, 256, 128)])
def test_tiles_of_eight_rows_are_as_exact_as_fp32(oracle, type_, rows, cols):
    w = formats.quantize(type_, synth.normal(81, (rows, cols), 0.02)).reshape(-1)
    t = dev(w)
    ms = L.matrix_set(t, type_, formats.GGUF, rows, cols, 1)
    x = synth.normal(83, (16, cols), 1.0)
    want = x.astype(np.float64) @ oracle.dequantize(type_, w, rows * cols).astype(np.float64).reshape(rows, cols).T
    dx = dev(x)
    e = torch.zeros(1, dtype=torch.int32, device=DEV)

    def error(T, n):
        out = torch.zeros((T, rows), dtype=torch.float32, device=DEV)
        capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, 1, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        return float(np.linalg.norm(out.cpu().numpy()[:n].astype(np.float64) - want[:n]) / np.linalg.norm(want[:n]))
    for T in (8, 3):   # low halves in a pass of their own; in the free columns
        assert error(T, T) <= error(16, T)
    assert int(e.item()) == 0


# An outlier that meets weights of zero (a block whose scale and offset are zero) leaves the other values as they are, however much larger it
# is: n * 2^-24 of the sum of the terms' own magnitudes, as FP32 sums give it. Either side of the limit from which a row takes FP32 sums.
@pytest.mark.parametrize("type_,rows,cols", [(formats.Q5_K, 16, 512), (formats.Q5_K, 144, 2048), (formats.Q5_1, 16, 128), (formats.Q5_1, 272, 512)])
@pytest.mark.parametrize("gate_up", [False, True])
def test_outliers_at_zero_weights(oracle, type_, rows, cols, gate_up):
    w = formats.quantize(type_, synth.normal(84, (rows, cols), 0.02)).reshape(rows, -1).copy()
    block, width = (176, 256) if type_ == formats.Q5_K else (24, 32)
    w[:, :block] = 0
    w = w.reshape(-1)
    t = dev(w)
    ms = L.matrix_set(t, type_, formats.GGUF, rows, cols, 1)
    w64 = oracle.dequantize(type_, w, rows * cols).astype(np.float64).reshape(rows, cols)
    assert not w64[:, :width].any()
    x = synth.normal(85, (8, cols), 1.0)
    for j in range(1, 8):
        x[j, 3] = 2.0 ** (0, 8, 13, 16, 24, 39, 60, 120)[j]
    x64 = x.astype(np.float64)
    want = x64 @ w64.T
    bound = (cols + 8) * 2.0 ** -24 * 4 * np.abs(w64).max() * np.abs(x64[:, width:]).sum(axis=1)[:, None]   # a term: see the tile edges above
    if gate_up:
        want, bound = want / (1 + np.exp(-want)) * want, bound * (2 * np.abs(want) + 2)
    dx, e = dev(x), torch.zeros(1, dtype=torch.int32, device=DEV)
    rows_of = {}
    for T in (8, 4):
        out = torch.zeros((T, rows), dtype=torch.float32, device=DEV)
        if gate_up:
            capi.call("tsp_moe_gate_up_swiglu", C.byref(ms), C.byref(ms), dx.data_ptr(), cols * 4, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        else:
            capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, 1, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        rows_of[T] = out.cpu().numpy()
        assert np.all(np.abs(rows_of[T] - want[:T]) <= bound[:T])
    assert np.array_equal(rows_of[4], rows_of[8][:4])
    assert int(e.item()) == 0


def test_every_kernel_gets_its_own_shared_memory_limit(oracle):
    """Dense batches of 16 rows: the plain kernel and the gate-up kernel of one encoding both need more than the default 48 KB of shared
    memory; the limit set for one says nothing about the other."""
    rows, cols, T = 16, 2048, 16
    w = formats.quantize(formats.Q5_K, synth.normal(91, (rows, cols), 0.02)).reshape(-1)
    t = dev(w)
    ms = L.matrix_set(t, formats.Q5_K, formats.GGUF, rows, cols, 1)
    x = synth.normal(92, (T, cols), 1.0)
    dx, e = dev(x), torch.zeros(1, dtype=torch.int32, device=DEV)
    out, h = (torch.zeros((T, rows), dtype=torch.float32, device=DEV) for _ in range(2))
    capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, 1, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
    capi.call("tsp_moe_gate_up_swiglu", C.byref(ms), C.byref(ms), dx.data_ptr(), cols * 4, T, 1, None, None, None, h.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert int(e.item()) == 0
    want = np.stack([oracle.gemv(formats.Q5_K, w, cols, rows, x[i]) for i in range(T)]).astype(np.float64)
    assert scaled_error(out.cpu().numpy(), want) <= 5e-5
    assert scaled_error(h.cpu().numpy(), want / (1 + np.exp(-want)) * want) <= 5e-5


@pytest.mark.parametrize("T", [1, 8, 29, 64])
@pytest.mark.parametrize("shared_type", [formats.Q8_0, formats.Q5_K])
def test_layer_q5k_gate_up_q51_down(oracle, T, shared_type):
    """The reference model's pairing: Q5_K gate / up, Q5_1 down, Q8_0 shared expert (and, as a second case, a Q5_K shared
    expert through the same plain kernel), top-4 of 16 experts so that tiles of more than 8 routes occur."""
    Cn, H, E, K = 512, 256, 16, 4
    q = formats.quantize
    ex = lambda s, t, r, c: np.stack([q(t, synth.normal(s * 1000 + e, (r, c), 0.02)).reshape(-1) for e in range(E)])
    host = L.HostLayer(Cn, H, E, K, formats.Q5_K, shared_type, ex(1, formats.Q5_K, H, Cn), ex(2, formats.Q5_K, H, Cn), ex(3, formats.Q5_1, Cn, H),
                       q(shared_type, synth.normal(7001, (H, Cn), 0.02)).reshape(-1), q(shared_type, synth.normal(7002, (H, Cn), 0.02)).reshape(-1),
                       q(shared_type, synth.normal(7003, (Cn, H), 0.02)).reshape(-1), synth.normal(7004, (Cn,), 0.02), down_type=formats.Q5_1)
    x16 = synth.activations_f16(5, T, Cn)
    logits = synth.router_logits(6, T, E)
    dl = L.DeviceLayer(host, formats.GGUF, DEV)
    s = L.Scratch(Cn, H, E, K, T, DEV)
    out = torch.zeros((T, Cn), dtype=torch.float32, device=DEV)
    L.moe_layer_decode(dl, s, dev(x16.astype(np.float32)), dev(logits), out)
    torch.cuda.synchronize()
    assert s.error_word() == 0
    want, st = oracle.moe_layer(host.oracle_dict(), x16.astype(np.float32), logits, threads=4, stages=True)
    assert np.array_equal(s.ids.cpu().numpy().view(np.uint32)[:T * K].reshape(T, K), st["indices"])
    assert scaled_error(s.hidden.cpu().numpy()[:T * K * H].reshape(T, K, H), st["activated"]) <= 5e-5
    assert scaled_error(s.routed.cpu().numpy()[:T * K * Cn].reshape(T, K, Cn), st["routed"]) <= 5e-5
    assert scaled_error(s.shared_out.cpu().numpy()[:T * Cn].reshape(T, Cn), st["shared_out"]) <= 5e-5
    assert scaled_error(out.cpu().numpy(), want) <= 5e-5


def test_nonfinite_scale_sets_the_error_word():
    w = formats.quantize(formats.Q5_1, synth.normal(61, (16, 64), 0.02)).reshape(-1).copy()
    w[0:2] = [0x00, 0x7c]   # d = +inf in the first block
    t = dev(w)
    ms = L.matrix_set(t, formats.Q5_1, formats.GGUF, 16, 64, 1)
    dx = dev(synth.normal(62, (1, 64), 1.0))
    out = torch.zeros((1, 16), dtype=torch.float32, device=DEV)
    e = torch.zeros(1, dtype=torch.int32, device=DEV)
    capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), 256, 1, 1, 1, None, None, None, out.data_ptr(), 64, 0, e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert int(e.item()) & capi.ERR_NONFINITE


# Infinities and NaN in a token row, on the MMA kernel's tiles (8 rows) and the FP32 kernel's (16): reported, and every other row as without them
@pytest.mark.parametrize("T", [3, 8, 16])
@pytest.mark.parametrize("type_,rows,cols", [(formats.Q5_K, 32, 512), (formats.Q5_1, 32, 128)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_nonfinite_activation_row(type_, rows, cols, T, bad):
    w = formats.quantize(type_, synth.normal(95, (rows, cols), 0.02)).reshape(-1)
    t = dev(w)
    ms = L.matrix_set(t, type_, formats.GGUF, rows, cols, 1)
    x = synth.normal(96, (T, cols), 1.0)
    outs = []
    for value in (x[1, 5], bad):
        x[1, 5] = value
        dx, out, e = dev(x), torch.zeros((T, rows), dtype=torch.float32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, 1, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        assert bool(int(e.item()) & capi.ERR_NONFINITE) == (not np.isfinite(value))
        outs.append(out.cpu().numpy())
    others = [i for i in range(T) if i != 1]
    assert np.array_equal(outs[0][others], outs[1][others])
    assert not np.isfinite(outs[1][1]).any()


@pytest.mark.parametrize("T", [1, 5])
def test_rows_do_not_depend_on_how_a_dense_launch_is_split(T):
    """Dense launches of 16, 2400, 4800 and 9616 rows take one, two, four and eight warps per block's item: a row comes out the same."""
    rows, cols = 9616, 128
    w = formats.quantize(formats.Q5_1, synth.normal(97, (rows, cols), 0.02)).reshape(rows, -1)
    dx, e, outs = dev(synth.normal(98, (T, cols), 1.0)), torch.zeros(1, dtype=torch.int32, device=DEV), []
    for n in (9616, 4800, 2400, 16):
        t = dev(w[:n].reshape(-1))
        ms = L.matrix_set(t, formats.Q5_1, formats.GGUF, n, cols, 1)
        out = torch.zeros((T, n), dtype=torch.float32, device=DEV)
        capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, 1, T, 1, None, None, None, out.data_ptr(), n * 4, 0, e.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        outs.append(out.cpu().numpy())
    assert int(e.item()) == 0
    for o in outs[1:]:
        assert np.array_equal(o, outs[0][:, :o.shape[1]])


# How the MMA kernel cuts its work: two warps per unit of rows with uneven parts (three steps of K), two, four and eight, two steps a warp (sixteen), rows whose
# unit takes two copies (more than 256 lines), a unit count that the blocks do not share evenly. An FP32 sum of n terms: see the tile edges above.
@pytest.mark.parametrize("type_,rows,cols", [(formats.Q5_K, 48, 768), (formats.Q5_K, 2400, 512), (formats.Q5_K, 32, 3072), (formats.Q5_1, 3008, 384), (formats.Q5_1, 48, 2944),
                                             (formats.Q5_1, 32, 2048),
                                             # enough units per block to go round the ring of stages: one, two and four warps per unit
                                             (formats.Q5_K, 47360, 256), (formats.Q5_K, 28416, 768), (formats.Q5_1, 47360, 128), (formats.Q5_1, 47360, 640)])
@pytest.mark.parametrize("gate_up", [False, True])
def test_unit_geometry(oracle, type_, rows, cols, gate_up):
    w = formats.quantize(type_, synth.normal(101, (rows, cols), 0.02)).reshape(-1)
    t = dev(w)
    ms = L.matrix_set(t, type_, formats.GGUF, rows, cols, 1)
    x = synth.normal(102, (7, cols), 1.0)
    w64 = oracle.dequantize(type_, w, rows * cols).astype(np.float64).reshape(rows, cols)
    want = x.astype(np.float64) @ w64.T
    bound = (cols + 8) * 2.0 ** -24 * 4 * np.abs(w64).max() * np.abs(x.astype(np.float64)).sum(axis=1)[:, None]
    if gate_up:
        want, bound = want / (1 + np.exp(-want)) * want, bound * (2 * np.abs(want) + 2)
    dx, e = dev(x), torch.zeros(1, dtype=torch.int32, device=DEV)
    for T in (7, 2):
        out = torch.full((T, rows), np.nan, dtype=torch.float32, device=DEV)
        if gate_up:
            capi.call("tsp_moe_gate_up_swiglu", C.byref(ms), C.byref(ms), dx.data_ptr(), cols * 4, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        else:
            capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, 1, T, 1, None, None, None, out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        assert np.all(np.abs(out.cpu().numpy() - want[:T]) <= bound[:T])
    assert int(e.item()) == 0


@pytest.mark.parametrize("tokens,experts,selected", [(1500, 512, 32), (2048, 4096, 32)])
def test_many_tiles_per_block(oracle, tokens, experts, selected):
    """Blocks that walk more tiles than their routing table holds (32), with the experts in two address ranges."""
    rows, cols = 16, 128
    rng = np.random.default_rng(7)
    w = rng.integers(0, 256, (experts, rows * cols // 32 * 24), dtype=np.uint8)
    w.reshape(experts, -1, 24)[:, :, 0:4] = np.array([0x00, 0x24, 0x00, 0xa4], dtype=np.uint8)   # d = 2^-6, m = -2^-6
    t = dev(w.reshape(-1))
    half = experts // 2
    ms = L.matrix_set(t, formats.Q5_1, formats.GGUF, rows, cols, experts, base_hi=t.reshape(experts, -1)[half:].reshape(-1), split=half)
    ids = np.argsort(rng.random((tokens, experts)), axis=1)[:, :selected].astype(np.int32)
    x = synth.normal(103, (tokens, cols), 1.0)
    dx, dids, e = dev(x), dev(ids), torch.zeros(1, dtype=torch.int32, device=DEV)
    tmap, counts = torch.empty(experts * tokens, dtype=torch.int32, device=DEV), torch.empty(experts, dtype=torch.int32, device=DEV)
    tasks = torch.empty(capi.lib().tsp_moe_tasks_words(tokens, experts, selected, 8), dtype=torch.int32, device=DEV)
    out = torch.full((tokens * selected, rows), np.nan, dtype=torch.float32, device=DEV)
    capi.call("tsp_moe_permute", dids.data_ptr(), tokens, experts, selected, 8, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(), e.data_ptr(), L.stream_ptr())
    capi.call("tsp_moe_project", C.byref(ms), dx.data_ptr(), cols * 4, selected, tokens, selected, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(),
              out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert int(e.item()) == 0
    # a unit of 16 rows per tile, spread evenly: every block has more tiles than its table
    assert int(tasks[0]) > 33 * torch.cuda.get_device_properties(0).multi_processor_count
    w64 = oracle.dequantize(formats.Q5_1, w.reshape(-1), experts * rows * cols).astype(np.float64).reshape(experts, rows, cols)
    want = np.einsum("tkrc,tc->tkr", w64[ids[::16]], x[::16].astype(np.float64))
    got = out.cpu().numpy().reshape(tokens, selected, rows)[::16]
    bound = (cols + 8) * 2.0 ** -24 * 4 * np.abs(w64).max() * np.abs(x[::16].astype(np.float64)).sum(axis=1)[:, None, None]
    assert np.isfinite(out.cpu().numpy()).all() and np.all(np.abs(got - want) <= bound)


# Short rows: whole blocks per tile where the tiles are fewer than the blocks (one block of several units, several blocks per tile and blocks without work
# at the end), an even split beyond; each row the bits it has alone
@pytest.mark.parametrize("tokens,experts,selected", [(8, 3, 1), (40, 16, 2), (64, 64, 4), (300, 100, 8), (8, 200, 40)])
@pytest.mark.parametrize("type_,rows,cols", [(formats.Q5_K, 256, 512), (formats.Q5_1, 272, 128), (formats.Q5_1, 64, 1024)])
@pytest.mark.parametrize("gate_up", [False, True])
def test_whole_blocks_per_tile(oracle, type_, rows, cols, gate_up, tokens, experts, selected):
    rng = np.random.default_rng(tokens + experts)
    w = np.concatenate([formats.quantize(type_, synth.normal(200 + i % 7, (rows, cols), 0.02)).reshape(-1) for i in range(experts)])
    t = dev(w)
    ms = L.matrix_set(t, type_, formats.GGUF, rows, cols, experts)
    ids = np.argsort(rng.random((tokens, experts)), axis=1)[:, :selected].astype(np.int32)
    dx, e = dev(synth.normal(104, (tokens, cols), 1.0)), torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(x, which):
        n = len(which)
        dids = dev(which)
        tmap, counts = torch.empty(experts * n, dtype=torch.int32, device=DEV), torch.empty(experts, dtype=torch.int32, device=DEV)
        tasks = torch.empty(capi.lib().tsp_moe_tasks_words(n, experts, selected, 8), dtype=torch.int32, device=DEV)
        out = torch.full((n * selected, rows), np.nan, dtype=torch.float32, device=DEV)
        capi.call("tsp_moe_permute", dids.data_ptr(), n, experts, selected, 8, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(), e.data_ptr(), L.stream_ptr())
        if gate_up:
            capi.call("tsp_moe_gate_up_swiglu", C.byref(ms), C.byref(ms), x.data_ptr(), cols * 4, n, selected, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(),
                      out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        else:
            capi.call("tsp_moe_project", C.byref(ms), x.data_ptr(), cols * 4, selected, n, selected, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(),
                      out.data_ptr(), rows * 4, 0, e.data_ptr(), L.stream_ptr())
        torch.cuda.synchronize()
        return out.view(n, selected, rows)

    got = run(dx, ids)
    assert int(e.item()) == 0 and bool(torch.isfinite(got).all())
    for at in range(0, tokens, max(1, tokens // 8)):   # one row: an even split
        assert torch.equal(run(dx[at:at + 1], ids[at:at + 1])[0], got[at])
