"""Decode batches of up to eight rows route inside the gate-up launch: ids, mixture weights and tables as the separate launches (tsp_moe_route,
tsp_moe_permute) and the oracle give them, the layer's rows as the tables of a larger batch give them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tokspur_public_b200 import capi, formats, synth  # noqa: E402
from tokspur_public_b200 import layer as L  # noqa: E402

DEV = "cuda"


def logits_of(kind, rows, experts, seed):
    l = synth.router_logits(seed, rows, experts)
    if kind == "ties":       # five distinct values: more logits reach the bound than a warp has lanes
        l = np.round(l).clip(-2, 2).astype(np.float32)
    elif kind == "zeros":    # -0 and +0 are one value, ties go to the lower id
        l[:, ::2] = 0.0
        l[:, 1::2] = -0.0
    elif kind == "lane":     # all winners in one lane of the selecting warp
        l[:, 3::32] += 100.0
    return l


@pytest.mark.parametrize("kind", ["normal", "ties", "zeros", "lane"])
@pytest.mark.parametrize("experts,selected", [(8, 8), (33, 10), (512, 1), (512, 8), (512, 9), (512, 10), (512, 32), (512, 33), (500, 64)])
@pytest.mark.parametrize("mode", [0, 1])
def test_selection_against_oracle(oracle, kind, experts, selected, mode):
    rows = 5
    logits = logits_of(kind, rows, experts, 31)
    dl = torch.from_numpy(logits).to(DEV)
    ids, w = torch.empty(rows * selected, dtype=torch.int32, device=DEV), torch.empty(rows * selected, device=DEV)
    e = torch.zeros(1, dtype=torch.int32, device=DEV)
    capi.call("tsp_moe_route", dl.data_ptr(), experts * 4, rows, experts, selected, mode, 1, ids.data_ptr(), w.data_ptr(), e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    want_ids, want_w = oracle.route_rows(logits, selected, mode, True)
    assert int(e.item()) == 0
    assert np.array_equal(ids.cpu().numpy().view(np.uint32).reshape(rows, selected), want_ids)
    assert np.allclose(w.cpu().numpy().reshape(rows, selected), want_w, rtol=2.0 ** -22, atol=2.0 ** -149)   # 64-bit weights rounded once (to a multiple of 2^-149)


@pytest.mark.parametrize("layout", [formats.PLANAR, formats.GGUF])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("channels,hidden,experts,selected,kind", [(1024, 256, 512, 10, "normal"), (2048, 256, 512, 64, "normal"), (1024, 256, 16, 4, "ties"), (1024, 256, 33, 33, "zeros")])
@pytest.mark.parametrize("tokens", [1, 3, 8])
def test_layer_routes_its_own_batch(layout, dtype, channels, hidden, experts, selected, kind, tokens):
    dl = L.SynthDeviceLayer(9, channels, hidden, experts, formats.Q4_K, layout, DEV)
    big = 24   # rows of a batch that takes the separate launches; its first `tokens` rows are the small batch
    x = torch.from_numpy(synth.normal(32, (big, channels), 1.0)).to(DEV).to(dtype)
    logits = torch.from_numpy(logits_of(kind, big, experts, 33)).to(DEV)
    outs = []
    for n in (tokens, big):
        s = L.Scratch(channels, hidden, experts, selected, n, DEV)
        for t in (s.ids, s.counts, s.tasks, s.token_map):
            t.fill_(-7)
        s.weights.fill_(float("nan"))
        out = torch.empty(n, channels, device=DEV)
        L.moe_layer_decode(dl, s, x[:n], logits[:n], out)
        torch.cuda.synchronize()
        assert s.error_word() == 0
        outs.append(out.cpu().numpy())
        if n == tokens:
            small = s
    # a row's sums do not depend on the tile it is in
    assert np.array_equal(outs[0], outs[1][:tokens])
    ids, w, e = torch.empty(tokens * selected, dtype=torch.int32, device=DEV), torch.empty(tokens * selected, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    tmap, counts = torch.full((experts * tokens,), -7, dtype=torch.int32, device=DEV), torch.empty(experts, dtype=torch.int32, device=DEV)
    words = int(capi.lib().tsp_moe_tasks_words(tokens, experts, selected, 8))
    tasks = torch.empty(words, dtype=torch.int32, device=DEV)
    capi.call("tsp_moe_route", logits.data_ptr(), experts * 4, tokens, experts, selected, 0, 1, ids.data_ptr(), w.data_ptr(), e.data_ptr(), L.stream_ptr())
    capi.call("tsp_moe_permute", ids.data_ptr(), tokens, experts, selected, 8, tmap.data_ptr(), counts.data_ptr(), tasks.data_ptr(), e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    for mine, want in ((small.ids, ids), (small.weights, w), (small.counts, counts), (small.tasks[:words], tasks), (small.token_map, tmap)):
        assert torch.equal(mine[:len(want)], want)


@pytest.mark.parametrize("tokens", [1, 8])
def test_nonfinite_logits_are_reported(tokens):
    channels, hidden, experts, selected = 1024, 256, 64, 4
    dl = L.SynthDeviceLayer(9, channels, hidden, experts, formats.Q4_K, formats.PLANAR, DEV)
    x, logits = torch.from_numpy(synth.normal(34, (tokens, channels), 1.0)).to(DEV), synth.router_logits(35, tokens, experts)
    outs = []
    for bad in (logits[tokens - 1, 7], np.nan):
        logits[tokens - 1, 7] = bad
        s, out = L.Scratch(channels, hidden, experts, selected, tokens, DEV), torch.empty(tokens, channels, device=DEV)
        L.moe_layer_decode(dl, s, x, torch.from_numpy(logits).to(DEV), out)
        torch.cuda.synchronize()
        assert bool(int(s.error.cpu()[0]) & capi.ERR_NONFINITE) == (not np.isfinite(bad))
        outs.append(out.cpu().numpy())
    assert np.array_equal(outs[0][:tokens - 1], outs[1][:tokens - 1])
    assert not s.weights.cpu().numpy()[(tokens - 1) * selected:tokens * selected].any()


def layer_rows(dl, shape, tokens, x, logits, out, share=None):
    """Output rows of one call; share(scratch): gives some of the scratch's pointers other buffers' memory."""
    s = L.Scratch(*shape, tokens, DEV)
    if share:
        share(s)
    L.moe_layer_decode(dl, s, x, logits, out)
    torch.cuda.synchronize()
    assert s.error_word() == 0
    return out.clone()


# Up to eight rows the mixture reads the caller's binary16 rows, in slices of a row; nine rows take the FP32 copy. `beside`: output rows between
# the input rows of one buffer
@pytest.mark.parametrize("tokens", [1, 8, 9])
@pytest.mark.parametrize("place", ["same", "shifted", "beside"])
def test_output_in_the_input_rows(tokens, place):
    shape = channels, hidden, experts, selected = 2048, 256, 16, 4
    dl = L.SynthDeviceLayer(9, channels, hidden, experts, formats.Q4_K, formats.PLANAR, DEV)
    rows = torch.from_numpy(synth.normal(36, (tokens, channels), 1.0)).to(DEV).half()
    logits = torch.from_numpy(synth.router_logits(37, tokens, experts)).to(DEV)
    want = layer_rows(dl, shape, tokens, rows, logits, torch.empty_like(rows))
    for _ in range(20):
        buf = torch.empty(tokens * 2 * channels + channels, dtype=torch.float16, device=DEV)
        if place == "beside":
            both = buf[:tokens * 2 * channels].view(tokens, 2 * channels)
            x, out = both[:, :channels], both[:, channels:]
        else:
            at = 8 if place == "shifted" else 0
            x, out = (buf[o:o + tokens * channels].view(tokens, channels) for o in (0, at))
        x.copy_(rows)
        assert torch.equal(layer_rows(dl, shape, tokens, x, logits, out), want)


# What one launch does now was done in turn by several: buffers that those did not need at the same time may be the same memory
@pytest.mark.parametrize("tokens", [3, 8])
@pytest.mark.parametrize("shared", ["rows in routed", "rows in shared_out", "ids in hidden", "logits in hidden", "logits in shared_hidden"])
def test_buffers_that_share_memory(tokens, shared):
    shape = channels, hidden, experts, selected = 1024, 256, 512, 10
    dl = L.SynthDeviceLayer(9, channels, hidden, experts, formats.Q4_K, formats.PLANAR, DEV)
    x = torch.from_numpy(synth.normal(38, (tokens, channels), 1.0)).to(DEV).half()
    logits = torch.from_numpy(synth.router_logits(39, tokens, experts)).to(DEV)
    want = layer_rows(dl, shape, tokens, x, logits, torch.empty_like(x))
    own, other = shared.split(" in ")
    room = torch.zeros(max(tokens * selected * channels, tokens * experts), device=DEV)
    if own == "rows":
        x = room.view(torch.float16)[:x.numel()].view_as(x).copy_(x)
    elif own == "logits":
        logits = room[:logits.numel()].view_as(logits).copy_(logits)

    def share(s):
        setattr(s.c, "d_" + other, room.data_ptr())
        if own == "ids":
            s.c.d_ids = room.data_ptr()

    assert torch.equal(layer_rows(dl, shape, tokens, x, logits, torch.empty_like(x), share), want)
