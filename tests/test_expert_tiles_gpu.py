"""The experts' products on tcgen05 at the borders of their dispatch: 16, 32 and 64 columns, narrow and wide tiles, an expert
with more rows than columns, matrices that fill no whole tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def k():
    from chibillm_b200.kernels.ops import CudaKernels
    return CudaKernels(torch.device(DEV))


# D, F: one K block; several, and 2 F and D beyond whole tiles of 128 and 256; two choices of a token may be one expert
@pytest.mark.parametrize("D,F", [(64, 64), (320, 192), (640, 320)])
@pytest.mark.parametrize("T,E,top,same", [(1, 4, 2, False), (12, 4, 2, True), (16, 8, 1, False), (17, 8, 2, False), (33, 3, 3, True),
                                          (64, 2, 1, False), (65, 8, 2, False), (130, 40, 2, False), (300, 4, 2, False),
                                          (1500, 5, 2, False)])
@pytest.mark.parametrize("weight_on_input", [False, True])
def test_chosen_experts_tiles(k, D, F, T, E, top, same, weight_on_input):
    g = torch.Generator(device=DEV).manual_seed(T + D)
    rnd = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=DEV) * std)
    x = rnd(T, D).bfloat16()
    gate, up, down = (rnd(E, a, b, std=b ** -0.5).bfloat16() for a, b in ((F, D), (F, D), (D, F)))
    if same:                                             # all choices the same expert
        chosen = torch.full((T, top), 1, dtype=torch.int32, device=DEV)
    else:
        chosen = torch.rand(T, E, generator=g, device=DEV).topk(top, 1).indices.to(torch.int32).contiguous()
    share = torch.rand(T, top, generator=g, device=DEV) + 0.1
    pairs = T * top
    out = torch.full((T, D), float("nan"), device=DEV)
    stacked = torch.stack([k.interleave_expert_gate_up(a, b) for a, b in zip(gate, up)]).contiguous()
    k.chosen_experts(x, chosen, share, stacked, down, out, torch.empty(k.route_words(pairs, E), dtype=torch.int32, device=DEV),
                     torch.empty(pairs, F, dtype=torch.bfloat16, device=DEV), torch.empty(pairs, D, device=DEV), "silu",
                     torch.empty(pairs, D, dtype=torch.bfloat16, device=DEV), gated=True, interleaved=True, overwrite=True,
                     weight_on_input=weight_on_input)
    k.check_error_word()
    ref, size = torch.zeros(T, D, dtype=torch.float64, device=DEV), torch.zeros(T, D, dtype=torch.float64, device=DEV)
    for s in range(top):
        e = chosen[:, s].long()
        w = share[:, s].double()[:, None]
        a = torch.einsum("td,tfd->tf", x.double(), gate.double()[e])
        b = torch.einsum("td,tfd->tf", x.double(), up.double()[e])
        if weight_on_input:
            a, b, w = w * a, w * b, torch.ones_like(w)
        act = torch.nn.functional.silu(a) * b
        ref += w * torch.einsum("tf,tdf->td", act, down.double()[e])
        size += w * torch.einsum("tf,tdf->td", act.abs(), down.double()[e].abs())
    # the activations become bfloat16 (half a unit of 2^-8) and the sums are 32-bit
    assert ((out.double() - ref).abs() <= (2.0 ** -9 * 1.1 + 1e-5) * size + 1e-6).all()


@pytest.mark.parametrize("T", [16, 64, 300])             # 16 and 64 columns, tiles of 128 rows
def test_the_gate_is_made_in_32_bits(k, T):
    """Products of one term each, so that the epilogue's arithmetic is all there is: the gate far into its tail too, where
    1 + exp(-z) is near the largest 32-bit number."""
    D = F = 64
    x = torch.eye(D, dtype=torch.bfloat16, device=DEV)[torch.arange(T, device=DEV) % D].contiguous()
    gate = torch.linspace(-88.0, 20.0, F * D, device=DEV).view(1, F, D).bfloat16()
    g = torch.Generator(device=DEV).manual_seed(1)
    up = (torch.randn(1, F, D, generator=g, device=DEV) * 2.0 ** 30).bfloat16()
    down = torch.eye(F, dtype=torch.bfloat16, device=DEV)[None].contiguous()
    out = torch.full((T, D), float("nan"), device=DEV)
    k.chosen_experts(x, torch.zeros(T, 1, dtype=torch.int32, device=DEV), torch.ones(T, 1, device=DEV),
                     k.interleave_expert_gate_up(gate[0], up[0])[None].contiguous(), down, out,
                     torch.empty(k.route_words(T, 1), dtype=torch.int32, device=DEV),
                     torch.empty(T, F, dtype=torch.bfloat16, device=DEV), torch.empty(T, D, device=DEV), "silu",
                     torch.empty(T, D, dtype=torch.bfloat16, device=DEV), gated=True, interleaved=True, overwrite=True)
    k.check_error_word()
    z, u = gate[0].double().t()[torch.arange(T, device=DEV) % D], up[0].double().t()[torch.arange(T, device=DEV) % D]
    ref = z * torch.sigmoid(z) * u
    # the rounding to bfloat16 (half a unit of the 8th significant bit: 2^-8 of a value at most) after an exponential of two
    # units in the last place, a sum, a division and a product (each half a unit of 2^-23)
    assert ((out.double() - ref).abs() <= (2.0 ** -8 + 8 * 2.0 ** -24) * ref.abs()).all()
