"""Kernel launches of a layer call: what the thread's counter shows, what tsp_moe_layer_*_launches say beforehand, and the numbers the documents give."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tokspur_public_b200 import capi, formats, synth  # noqa: E402
from tokspur_public_b200 import layer as L  # noqa: E402

DEV = "cuda"


def run(path, dl, channels, hidden, experts, selected, tokens, dtype, normalize):
    s = (L.Scratch if path == "decode" else L.PrefillScratch)(channels, hidden, experts, selected, tokens, DEV)
    x = torch.from_numpy(synth.normal(1, (tokens, channels), 1.0)).to(DEV).to(dtype)
    logits = torch.from_numpy(synth.router_logits(2, tokens, experts)).to(DEV)
    out = torch.zeros(tokens, channels, device=DEV)
    lib = capi.lib()
    before = lib.tsp_launch_count()
    if path == "decode":
        said = lib.tsp_moe_layer_decode_launches(C.byref(dl.weights), int(dtype == torch.float16), tokens, channels, hidden, experts, selected, 0, normalize)
    else:
        said = lib.tsp_moe_layer_prefill_launches(C.byref(dl.weights), tokens, experts, normalize)
    torch.cuda.synchronize()
    assert lib.tsp_launch_count() == before and not out.any()   # asking launches nothing
    (L.moe_layer_decode if path == "decode" else L.moe_layer_prefill)(dl, s, x, logits, out, normalize=bool(normalize))
    made = lib.tsp_launch_count() - before
    torch.cuda.synchronize()
    assert (s if path == "decode" else s.base).error_word() == 0
    return said, made


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("path,types,experts,tokens,normalize,want", [
    ("decode", (formats.Q4_K,) * 3, 16, 1, 1, 3), ("decode", (formats.Q4_K,) * 3, 16, 8, 1, 3), ("decode", (formats.Q4_K,) * 3, 16, 8, 0, 5),
    ("decode", (formats.Q4_K,) * 3, 16, 9, 1, 5), ("decode", (formats.Q4_K,) * 3, 600, 8, 1, 5), ("decode", (formats.Q8_0,) * 3, 16, 5, 1, 5),
    ("decode", (formats.Q5_K, formats.Q5_1, formats.Q8_0), 16, 13, 1, 5), ("decode", (formats.Q5_K, formats.Q5_1, formats.Q8_0), 16, 129, 1, 7),
    ("prefill", (formats.Q4_K,) * 3, 16, 160, 1, 7), ("prefill", (formats.Q4_K,) * 3, 16, 257, 1, 6), ("prefill", (formats.Q4_K, formats.Q4_K, formats.Q8_0), 16, 300, 1, 8),
    ("prefill", (formats.Q4_K,) * 3, 600, 300, 1, 7), ("prefill", (formats.Q4_K,) * 3, 16, 300, 0, 7)])
def test_launches_of_a_layer(path, types, experts, tokens, normalize, want, dtype):
    channels, hidden, selected = 1024, 256, 4
    layout = formats.PLANAR if types[0] == formats.Q4_K else formats.GGUF
    dl = L.SynthDeviceLayer(3, channels, hidden, experts, types[0], layout, DEV, down_type=types[1], shared_type=types[2])
    assert run(path, dl, channels, hidden, experts, selected, tokens, dtype, normalize) == (want, want)


def test_refused_layer_has_no_launches():
    dl = L.SynthDeviceLayer(3, 1024, 256, 16, formats.Q4_K, formats.PLANAR, DEV)
    assert capi.lib().tsp_moe_layer_decode_launches(C.byref(dl.weights), 0, 1, 1024, 256, 16, 17, 0, 1) == 0   # more selected than experts
    assert capi.lib().tsp_moe_layer_prefill_launches(C.byref(dl.weights), 0, 16, 1) == 0
