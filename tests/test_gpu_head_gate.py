"""The kernel that ends the recurrent mixers: heads divided by their root mean square, times a gain and a gate."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("size,heads", [(1, 3), (20, 3), (32, 1), (36, 5), (64, 32), (128, 7), (132, 2), (256, 3), (260, 2)])
@pytest.mark.parametrize("shift", [0, 1])
def test_head_norm_gate_at_every_width(size, heads, dtype, shift):
    """Heads of one and two pieces a lane, sizes that are no whole pieces or above the vector form's largest, views that are
    not aligned; shared and whole gains, both gates, denominators."""
    from cloud_inference_from_scratch_b200.engine.runtime import Runtime

    rt = Runtime("cuda:0", dtype)
    generator = torch.Generator().manual_seed(size)
    rand = lambda *shape: torch.randn(*shape, generator=generator)  # noqa: E731
    for tokens in (1, 17):
        o, gate = rand(tokens, heads * size + 4), rand(tokens, heads * size + 4)
        o_view, gate_view = o.cuda()[:, shift:shift + heads * size], gate.cuda()[:, shift:shift + heads * size]
        below = rand(tokens, heads).abs() + 0.5
        for shared, act, denominators in ((False, "sigmoid", None), (True, "silu", None), (False, "silu", below)):
            gain = rand(size if shared else heads * size)
            out = torch.full((tokens + 1, heads * size), 7.0, dtype=rt.dtype).cuda()
            rt.ops.head_norm_gate(o_view, gate_view, gain.cuda(), 1e-6, out[:tokens], heads, gate_act=act,
                                  denominators=None if denominators is None else denominators.cuda())
            x = o[:, shift:shift + heads * size].double().view(tokens, heads, size)
            if denominators is not None:
                x = x / denominators.double().unsqueeze(-1)
            z = gate[:, shift:shift + heads * size].double()
            scale = gain.double().repeat(heads) if shared else gain.double()
            want = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)).flatten(1) * scale
            want = want * torch.sigmoid(z) * (z if act == "silu" else 1.0)
            bound = 1e-5 if dtype == "float32" else 2.0 ** -8
            assert float((out[:tokens].double().cpu() - want).abs().max()) <= bound * float(want.abs().max())
            assert float((out[tokens] - 7.0).abs().max()) == 0
