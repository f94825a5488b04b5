"""Prefill-size path (grouped tcgen05 GEMMs) against the CPU oracle: hidden rows and routed rows per stage, then whole layers
with skewed expert loads, empty experts, partial tiles and experts with more than one tile of 128 routes.
Bar: rel-L2 <= 2e-3 (binary16 operands, FP32 accumulate); the reference's own bound for this path is NMSE 2e-3."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tokspur_public_b200 import capi, formats, synth  # noqa: E402
from tokspur_public_b200 import layer as L  # noqa: E402


def rel_l2(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("T,E,K,skew", [(3, 4, 2, False), (40, 4, 2, False), (200, 8, 3, True), (700, 8, 2, True), (1300, 4, 1, True)])
def test_prefill_layer_against_oracle(oracle, T, E, K, skew):
    Cn, H = 256, 256
    host = L.synth_host_layer(5, Cn, H, E, K, expert_type=formats.Q4_K)
    dl = L.DeviceLayer(host, formats.PLANAR, "cuda")
    ps = L.PrefillScratch(Cn, H, E, K, T, "cuda")
    x16 = synth.activations_f16(7, T, Cn)
    logits = synth.router_logits(8, T, E, synth.zipf_bias(9, E) * 3 if skew else None)
    x32 = torch.from_numpy(x16.astype(np.float32)).cuda()
    out = torch.zeros((T, Cn), dtype=torch.float32, device="cuda")
    L.moe_layer_prefill(dl, ps, x32, torch.from_numpy(logits).cuda(), out)
    torch.cuda.synchronize()
    assert ps.base.error_word() == 0
    n = min(T, 24)
    sample = np.unique(np.linspace(0, T - 1, n).astype(int))
    want, st = oracle.moe_layer(host.oracle_dict(), x16[sample].astype(np.float32), logits[sample], threads=4, stages=True)
    ids = ps.base.ids.cpu().numpy().view(np.uint32)[:T * K].reshape(T, K)
    assert np.array_equal(ids[sample], st["indices"])
    routed = ps.routed_rows(T).reshape(T, K, Cn)
    assert rel_l2(routed[sample], st["routed"]) <= 2e-3
    shared = ps.shared_out_rows(T)
    assert rel_l2(shared[sample], st["shared_out"]) <= 2e-3
    assert rel_l2(out.cpu().numpy()[sample], want) <= 2e-3


@pytest.mark.parametrize("T,E,K,Cn,H,order", [(40, 4, 2, 256, 256, "separate"), (700, 8, 2, 512, 256, "gate_first"), (300, 3, 2, 256, 512, "up_first")])
def test_prefill_layer_gguf_blocks_against_oracle(oracle, T, E, K, Cn, H, order):
    """The same layer with the expert and shared tensors left as plain GGUF super-blocks (no planar copy): the code and header
    maps walk the 144-byte blocks. `order` puts gate and up in one allocation (one copy brings both when up follows gate at a
    constant distance) or the other way round (two copies), or leaves them as separate allocations."""
    host = L.synth_host_layer(11, Cn, H, E, K, expert_type=formats.Q4_K)
    dl = L.DeviceLayer(host, formats.GGUF, "cuda")
    if order != "separate":
        pair = np.concatenate([host.gate.reshape(-1), host.up.reshape(-1)] if order == "gate_first" else [host.up.reshape(-1), host.gate.reshape(-1)])
        both = torch.from_numpy(pair).cuda()
        dl.tensors.append(both)
        n = host.gate.size
        g_off, u_off = (0, n) if order == "gate_first" else (n, 0)
        dl.weights.gate = L.matrix_set(both, formats.Q4_K, formats.GGUF, H, Cn, E, offset=g_off)
        dl.weights.up = L.matrix_set(both, formats.Q4_K, formats.GGUF, H, Cn, E, offset=u_off)
    ps = L.PrefillScratch(Cn, H, E, K, T, "cuda")
    x16 = synth.activations_f16(12, T, Cn)
    logits = synth.router_logits(13, T, E, synth.zipf_bias(14, E) * 2)
    x32 = torch.from_numpy(x16.astype(np.float32)).cuda()
    out = torch.zeros((T, Cn), dtype=torch.float32, device="cuda")
    L.moe_layer_prefill(dl, ps, x32, torch.from_numpy(logits).cuda(), out)
    torch.cuda.synchronize()
    assert ps.base.error_word() == 0
    sample = np.unique(np.linspace(0, T - 1, 24).astype(int))
    want, st = oracle.moe_layer(host.oracle_dict(), x16[sample].astype(np.float32), logits[sample], threads=4, stages=True)
    routed = ps.routed_rows(T).reshape(T, K, Cn)
    assert rel_l2(routed[sample], st["routed"]) <= 2e-3
    assert rel_l2(ps.shared_out_rows(T)[sample], st["shared_out"]) <= 2e-3
    assert rel_l2(out.cpu().numpy()[sample], want) <= 2e-3
    # the planar copy of the same weights gives the same bits: both layouts stage identical binary16 operands
    dp = L.DeviceLayer(host, formats.PLANAR, "cuda")
    out_p = torch.zeros_like(out)
    L.moe_layer_prefill(dp, ps, x32, torch.from_numpy(logits).cuda(), out_p)
    torch.cuda.synchronize()
    assert torch.equal(out, out_p)


def test_staged_weight_values_against_rounded_reference(oracle):
    """The binary16 weight values the tensor-core kernels multiply, against RN16 of the reference's dequantised value.
    The kernels stage RN16((q - 8) * RN16(d*sc) + RN16(8*d*sc - dmin*mn)): three roundings of small quantities instead of one
    rounding of the exact value. Bound checked here: relative L2 deviation from the exact values <= 4e-4 (one rounding alone
    gives about 2.1e-4), no value further than 2^-10 of its group's largest magnitude from the once-rounded value."""
    rows, cols = 128, 2048
    w = formats.quantize_q4_k(synth.normal(17, (rows, cols), 0.02)).reshape(-1)
    planar = formats.pack_planar(formats.Q4_K, w, rows, cols)
    t = torch.from_numpy(planar).cuda()
    ms = L.matrix_set(t, formats.Q4_K, formats.PLANAR, rows, cols, 1)
    out = torch.zeros((rows, cols), dtype=torch.float16, device="cuda")
    capi.call("tsp_moe_staged_f16", C.byref(ms), 0, out.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    got = out.cpu().numpy().astype(np.float64)
    exact = oracle.dequantize(formats.Q4_K, w, rows * cols).reshape(rows, cols).astype(np.float64)
    once = exact.astype(np.float16).astype(np.float64)
    rel = np.linalg.norm(got - exact) / np.linalg.norm(exact)
    rel_once = np.linalg.norm(once - exact) / np.linalg.norm(exact)
    group_max = np.abs(exact).reshape(rows, cols // 32, 32).max(axis=2, keepdims=True)
    dev = (np.abs(got - once).reshape(rows, cols // 32, 32) / np.maximum(group_max, 1e-30)).max()
    print(f"staged weights: rel-L2 vs exact {rel:.3e} (one rounding: {rel_once:.3e}), worst deviation from RN16 {dev:.3e} of the group maximum")
    assert rel <= 4e-4 and dev <= 2.0 ** -10


def test_overflowing_hidden_row_is_reported_and_stays_alone(oracle):
    """Finite input rows whose hidden values pass binary16's range (the gate-up epilogue's test, with the columns past an expert's last route
    holding other experts' rows): reported; every other token row comes out as without them. One step below, nothing is reported."""
    Cn, H, E, K, T = 256, 256, 4, 2, 150
    host = L.synth_host_layer(23, Cn, H, E, K, expert_type=formats.Q4_K)
    x16, logits = synth.activations_f16(24, T, Cn), synth.router_logits(25, T, E)
    outs = []
    for scale in (1.0, 64.0, 16384.0):   # hidden values of the row about 0.1, 400 and 3e7
        x = x16.copy()
        x[77] = (x[77].astype(np.float32) * scale).clip(-60000, 60000).astype(np.float16)
        assert np.isfinite(x).all()
        dl = L.DeviceLayer(host, formats.PLANAR, "cuda")
        ps = L.PrefillScratch(Cn, H, E, K, T, "cuda")
        out = torch.zeros((T, Cn), dtype=torch.float32, device="cuda")
        L.moe_layer_prefill(dl, ps, torch.from_numpy(x.astype(np.float32)).cuda(), torch.from_numpy(logits).cuda(), out)
        torch.cuda.synchronize()
        assert bool(ps.base.error_word() & capi.ERR_NONFINITE) == (scale > 1000)
        outs.append(out.cpu().numpy())
    others = np.arange(T) != 77
    assert np.array_equal(outs[0][others], outs[1][others]) and np.array_equal(outs[0][others], outs[2][others])
    assert np.isfinite(outs[1]).all() and not np.isfinite(outs[2][77]).all()


# The cluster that builds the tables of more than 256 rows: an eighth of the rows per block in words of 32 (blocks without rows at 257), one word
# per block and several, the largest batch whose masks fit and the first that takes a block per pair of experts, an owner's slice of the experts
@pytest.mark.parametrize("tokens,experts,selected,first,local", [(257, 512, 10, 0, 512), (512, 512, 1, 0, 512), (1003, 1000, 8, 0, 1000), (2049, 16, 16, 0, 16), (4096, 512, 10, 128, 64),
                                                                 (16640, 512, 2, 0, 512), (16641, 512, 2, 0, 512), (300, 1024, 64, 0, 1024),
                                                                 (300, 8, 3, 0, 8), (549, 8, 2, 0, 8), (550, 8, 2, 0, 8), (639, 8, 1, 0, 8), (640, 8, 1, 0, 8)])   # few routes: one block
def test_tables_of_large_batches(oracle, tokens, experts, selected, first, local):
    rng = np.random.default_rng(tokens)
    ids = np.argsort(rng.random((tokens, experts), dtype=np.float32) - (np.arange(experts) < experts // 8) * 0.5, axis=1)[:, :selected].astype(np.uint32)
    dids = torch.from_numpy(ids.view(np.int32)).cuda()
    tmap, counts = torch.full((local * tokens,), -7, dtype=torch.int32, device="cuda"), torch.empty(local, dtype=torch.int32, device="cuda")
    words = int(capi.lib().tsp_moe_tasks_words(tokens, local, selected, 32))
    tasks, e = torch.full((words,), -7, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    if local == experts:
        capi.call("tsp_moe_permute", dids.data_ptr(), tokens, experts, selected, 32, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(), e.data_ptr(), L.stream_ptr())
    else:
        capi.call("tsp_moe_permute_local", dids.data_ptr(), tokens, first, local, selected, 32, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(), e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert int(e.item()) == 0
    want_counts = np.bincount(ids.reshape(-1), minlength=experts)[first:first + local]
    assert np.array_equal(counts.cpu().numpy(), want_counts)
    order = np.argsort(ids.reshape(-1), kind="stable")   # routes by expert, ascending
    starts = np.concatenate([[0], np.cumsum(np.bincount(ids.reshape(-1), minlength=experts))])
    got = tmap.cpu().numpy().reshape(local, tokens)
    for i in range(local):
        n = want_counts[i]
        assert np.array_equal(got[i, :n], order[starts[first + i]:starts[first + i] + n]) and (got[i, n:] == -7).all()
    pairs = [(i, t) for i in range(local) for t in range(0, want_counts[i], 32)]
    want_tasks = np.full(words, 0xffffffff, dtype=np.uint32)
    want_tasks[:2 + 2 * len(pairs)] = np.array([len(pairs), want_counts.sum()] + [v for p in pairs for v in p], dtype=np.uint32)
    assert np.array_equal(tasks.cpu().numpy().view(np.uint32), want_tasks)


# Few experts: slices of up to 65536 rows per block of the cluster, all of one expert's (the running counts are 16 bits), and the first batch beyond
@pytest.mark.parametrize("tokens", [524288, 524289, 600000])
@pytest.mark.parametrize("experts", [1, 16])
def test_tables_of_very_large_batches(tokens, experts):
    selected = 1 if experts == 1 else 2
    ids = np.zeros((tokens, selected), dtype=np.int32)   # every row names expert 0
    ids[:, 1:] = 1 + np.random.default_rng(tokens).integers(0, max(experts - 1, 1), (tokens, selected - 1))
    dids, e = torch.from_numpy(ids).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
    tmap, counts = torch.full((experts * tokens,), -7, dtype=torch.int32, device="cuda"), torch.empty(experts, dtype=torch.int32, device="cuda")
    tasks = torch.empty(int(capi.lib().tsp_moe_tasks_words(tokens, experts, selected, 256)), dtype=torch.int32, device="cuda")
    capi.call("tsp_moe_permute", dids.data_ptr(), tokens, experts, selected, 256, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(), e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert int(e.item()) == 0
    want_counts = np.bincount(ids.reshape(-1), minlength=experts)
    assert np.array_equal(counts.cpu().numpy(), want_counts)
    got = tmap.cpu().numpy().reshape(experts, tokens)
    for i in range(experts):
        assert np.array_equal(got[i, :want_counts[i]], np.flatnonzero(ids.reshape(-1) == i)) and (got[i, want_counts[i]:] == -7).all()


@pytest.mark.parametrize("bad", ["twice", "range"])
def test_tables_of_large_batches_report_bad_ids(bad):
    tokens, experts, selected = 700, 64, 4
    ids = np.tile(np.arange(selected, dtype=np.int32), (tokens, 1))
    ids[650, 2] = ids[650, 1] if bad == "twice" else experts
    dids, e = torch.from_numpy(ids).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
    tmap, counts = torch.empty(experts * tokens, dtype=torch.int32, device="cuda"), torch.empty(experts, dtype=torch.int32, device="cuda")
    tasks = torch.empty(int(capi.lib().tsp_moe_tasks_words(tokens, experts, selected, 8)), dtype=torch.int32, device="cuda")
    capi.call("tsp_moe_permute", dids.data_ptr(), tokens, experts, selected, 8, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(), e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert int(e.item()) & capi.ERR_INDEX


# Without a shared router nothing reads the input rows after their K-ordered copy, and nothing the ids after the route tables. Rows: the last ones, of more
# blocks than run at a time
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("tokens,own,other", [(8192, "ids", "rows"), (8192, "weights", "rows"), (300, "ids", "offsets"), (1100, "ids", "offsets"), (1100, "ids", "tasks")])
def test_layer_buffers_that_share_memory(dtype, tokens, own, other):
    channels, hidden, experts, selected = 256, 256, 8, 2
    dl = L.SynthDeviceLayer(13, channels, hidden, experts, formats.Q4_K, formats.PLANAR, "cuda")
    dl.weights.d_shared_router = None
    x = torch.from_numpy(synth.activations_f16(14, tokens, channels)).cuda().to(dtype)
    logits = torch.from_numpy(synth.router_logits(15, tokens, experts)).cuda()
    outs = []
    for share in (False, True):
        ps, out = L.PrefillScratch(channels, hidden, experts, selected, tokens, "cuda"), torch.empty((tokens, channels), device="cuda")
        rows = x.clone()
        if share:
            room = torch.zeros(tokens * channels, device="cuda")
            setattr(ps.c.base, "d_" + own, room.data_ptr() + (x.numel() * x.element_size() - tokens * selected * 4 if other == "rows" else 0))
            if other == "rows":
                rows = room.view(dtype)[:x.numel()].view_as(x).copy_(x)
            elif other == "tasks":
                ps.c.base.d_tasks = room.data_ptr()
            else:
                ps.c.d_offsets = room.data_ptr()
        L.moe_layer_prefill(dl, ps, rows, logits, out)
        torch.cuda.synchronize()
        assert ps.base.error_word() == 0
        outs.append(out)
    assert torch.equal(outs[0], outs[1])


# In place: every block of the mixture that works on a part of a row reads the whole input row for the shared router
@pytest.mark.parametrize("path", ["decode", "prefill"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("tokens", [5, 64, 591, 592])
def test_layer_in_place(path, dtype, tokens):
    channels, hidden, experts, selected = 2048, 256, 8, 2
    dl = L.SynthDeviceLayer(13, channels, hidden, experts, formats.Q4_K, formats.PLANAR, "cuda")
    x = torch.from_numpy(synth.activations_f16(14, tokens, channels)).cuda().to(dtype)
    logits = torch.from_numpy(synth.router_logits(15, tokens, experts)).cuda()
    s = (L.Scratch if path == "decode" else L.PrefillScratch)(channels, hidden, experts, selected, tokens, "cuda")
    call = L.moe_layer_decode if path == "decode" else L.moe_layer_prefill
    want = torch.empty_like(x)
    call(dl, s, x, logits, want)
    for _ in range(20):
        rows = x.clone()
        call(dl, s, rows, logits, rows)
        assert torch.equal(rows, want)
