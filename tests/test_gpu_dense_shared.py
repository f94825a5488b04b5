"""The dense Q8_0 shared expert of a decode batch, worked on in the launches that route the batch and build its tables, against launches of its own
(tsp_moe_gate_up_swiglu / tsp_moe_project on the dense sets) and 64-bit sums."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tokspur_public_b200 import capi, formats, synth  # noqa: E402
from tokspur_public_b200 import layer as L  # noqa: E402

DEV = "cuda"


def layer(channels, hidden, experts=8, selected=2):
    dl = L.SynthDeviceLayer(3, channels, hidden, experts, formats.Q5_K, formats.GGUF, DEV, shared_type=formats.Q8_0, down_type=formats.Q5_1)
    return dl, experts, selected


def error_of(got, want):
    return float(np.linalg.norm(got.astype(np.float64) - want) / np.linalg.norm(want))


# One run of 256 columns per row, three, four and eight (one, two, four and eight warps per group of rows); a tile of eight rows, its edges, the last
# batch that takes this path and the first that does not
@pytest.mark.parametrize("channels,hidden", [(256, 256), (768, 512), (1024, 256), (2048, 512)])
@pytest.mark.parametrize("tokens", [1, 8, 9, 128, 129])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_against_its_own_launches(oracle, channels, hidden, tokens, dtype):
    dl, experts, selected = layer(channels, hidden)
    s = L.Scratch(channels, hidden, experts, selected, tokens, DEV)
    x = torch.from_numpy(synth.normal(5, (tokens, channels), 1.0)).to(DEV).to(dtype)
    logits = torch.from_numpy(synth.router_logits(6, tokens, experts)).to(DEV)
    out = torch.empty(tokens, channels, device=DEV)
    s.shared_out.fill_(float("nan"))
    L.moe_layer_decode(dl, s, x, logits, out)
    got = s.shared_out[:tokens * channels].reshape(tokens, channels).cpu().numpy()
    x32, h, own = x.float(), torch.empty(tokens, hidden, device=DEV), torch.empty(tokens, channels, device=DEV)
    e, w = torch.zeros(1, dtype=torch.int32, device=DEV), dl.weights
    capi.call("tsp_moe_gate_up_swiglu", C.byref(w.shared_gate), C.byref(w.shared_up), x32.data_ptr(), channels * 4, tokens, 1, None, None, None, h.data_ptr(), hidden * 4,
              int(dtype == torch.float16), e.data_ptr(), L.stream_ptr())
    capi.call("tsp_moe_project", C.byref(w.shared_down), h.data_ptr(), hidden * 4, 1, tokens, 1, None, None, None, own.data_ptr(), channels * 4, 0, e.data_ptr(), L.stream_ptr())
    torch.cuda.synchronize()
    assert s.error_word() == 0 and int(e.item()) == 0
    dense = [oracle.dequantize(formats.Q8_0, dl.gguf[n].cpu().numpy(), hidden * channels).astype(np.float64) for n in ("shared_gate", "shared_up", "shared_down")]
    x64 = x32.cpu().numpy().astype(np.float64)
    g, u = x64 @ dense[0].reshape(hidden, channels).T, x64 @ dense[1].reshape(hidden, channels).T
    want = (g / (1 + np.exp(-g)) * u) @ dense[2].reshape(channels, hidden).T
    # no further from 64 bits than the general path (the same call past 128 rows); both are FP32 sums of exact terms and 22-bit activations
    assert error_of(got, want) <= error_of(own.cpu().numpy(), want) * 1.05


@pytest.mark.parametrize("bad", [np.inf, np.nan, 1e6])   # binary16's range is the range of activations beside Q8_0 weights
def test_values_beyond_binary16_are_reported(bad):
    channels, hidden, tokens = 512, 256, 5
    dl, experts, selected = layer(channels, hidden)
    s = L.Scratch(channels, hidden, experts, selected, tokens, DEV)
    x = synth.normal(7, (tokens, channels), 1.0)
    logits, out = torch.from_numpy(synth.router_logits(8, tokens, experts)).to(DEV), torch.empty(tokens, channels, device=DEV)
    rows = []
    for value in (x[2, 77], bad):
        x[2, 77] = value
        s.reset_error()
        L.moe_layer_decode(dl, s, torch.from_numpy(x).to(DEV), logits, out)
        torch.cuda.synchronize()
        word = torch.zeros(1, dtype=torch.int32)
        word.copy_(s.error)
        assert bool(int(word.item()) & capi.ERR_NONFINITE) == (abs(value) > 65504 or not np.isfinite(value))
        rows.append(s.shared_out[:tokens * channels].reshape(tokens, channels).cpu().numpy())
    assert np.array_equal(rows[0][[0, 1, 3, 4]], rows[1][[0, 1, 3, 4]])


# The shared expert is worked on before the routed experts now; its output rows came last before, when most scratch was no longer needed, and its
# hidden rows after the routing. Buffers that share memory on those grounds (without a shared router nothing reads the input rows after gate-up)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("shared", ["shared_out in hidden", "shared_out in x32", "shared_out in rows", "shared_out in ids", "shared_hidden in ids", "shared_hidden in logits"])
def test_buffers_that_share_memory(dtype, shared):
    channels, hidden, tokens = 512, 256, 5
    dl, experts, selected = layer(channels, hidden)
    dl.weights.d_shared_router = None
    x = torch.from_numpy(synth.normal(9, (tokens, channels), 1.0)).to(DEV).to(dtype)
    logits = torch.from_numpy(synth.router_logits(10, tokens, experts)).to(DEV)
    outs = []
    for own, other in ((None, None), shared.split(" in ")):
        s, out = L.Scratch(channels, hidden, experts, selected, tokens, DEV), torch.empty(tokens, channels, device=DEV)
        room = torch.zeros(tokens * channels * selected, device=DEV)
        xr, lr = x, logits
        if own:
            setattr(s.c, "d_" + own, room.data_ptr())
        if other == "rows":
            xr = room.view(dtype)[:x.numel()].view_as(x).copy_(x)
        elif other == "logits":
            lr = room[:logits.numel()].view_as(logits).copy_(logits)
        elif other:
            setattr(s.c, "d_" + other, room.data_ptr())
        L.moe_layer_decode(dl, s, xr, lr, out)
        torch.cuda.synchronize()
        assert s.error_word() == 0
        outs.append(out)
    # the shared expert's sums are in another order in launches of its own; 22-bit activations, FP32 sums
    assert float((outs[0] - outs[1]).norm() / outs[0].norm()) < 2e-6
