"""Un-quantised experts of a prompt portion (csrc/experts_gemm.cu: bf16, grouped tensor-core GEMMs over the pairs sorted by expert) at the edges of their tiles,
against plain torch in 64 bits on the same bf16 operands.  Only the activations are rounded in between (2^-9 each): 2^-8 of sum_j |w_j| |W_down| |a_j| covers
that and the fp32 sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (tokens, width, ff, experts, choices): rows around 128 and 256 per expert, column tiles of 128 and 256 with remainders, K below one step of 64, one
# expert, an expert without rows, more experts than the tile list's first warp
@pytest.mark.parametrize("T,width,ff,E,top", [(128, 64, 128, 1, 1), (129, 264, 136, 3, 2), (300, 8, 520, 2, 1), (257, 512, 8, 4, 3), (48, 1000, 248, 40, 4), (1000, 256, 384, 5, 2)])
@pytest.mark.parametrize("kind", ["silu", "gelu_tanh", "clamped_glu", "relu2"])
def test_prompt_experts(T, width, ff, E, top, kind):
    from ktransformers_b200.operators.experts import KExpertsDense
    g = torch.Generator(device="cuda").manual_seed(T + ff)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    op = KExpertsDense(width, ff, E, gated=kind != "relu2", act=kind if kind != "relu2" else "silu", limit=1.5)
    for p, k in ((op.gate, width), (op.up, width), (op.down, ff)):
        if p is not None:
            p.data.copy_(rnd(*p.shape) * k ** -0.5)
    x, w = rnd(T, width).to(torch.bfloat16), 0.2 + torch.rand((T, top), generator=g, device="cuda")
    ids = torch.stack([torch.randperm(E + 2, generator=g, device="cuda")[:top] for _ in range(T)])      # two of them name no expert
    if E > 2:
        ids[ids == 1] = E + 5
    for on_input in (False, True):
        assert op._sorted_gemms(x, ids, w)
        got = op.forward_grouped(x, ids, w, on_input).double()
        want, room = torch.zeros_like(got), torch.zeros_like(got)
        for e in range(E):
            t, j = (ids == e).nonzero(as_tuple=True)
            wt = w[t, j].double().unsqueeze(1)
            i, o = (wt, torch.ones_like(wt)) if on_input else (torch.ones_like(wt), wt)
            u = x[t].double() @ op.up[e].double().T * i
            z = x[t].double() @ op.gate[e].double().T * i if op.gated else None
            if kind == "relu2":
                a = u.clamp(min=0) ** 2
            elif kind == "clamped_glu":
                z, u = z.clamp(max=1.5), u.clamp(-1.5, 1.5)
                a = z * torch.sigmoid(1.702 * z) * (u + 1)
            else:
                a = (torch.nn.functional.silu(z) if kind == "silu" else torch.nn.functional.gelu(z, approximate="tanh")) * u
            want.index_add_(0, t, o * (a @ op.down[e].double().T))
            room.index_add_(0, t, o * (a.abs() @ op.down[e].double().abs().T))
        assert ((got - want).abs() <= 2.0 ** -8 * room + 1e-6).all(), ((got - want).abs() / (room + 1e-6)).max().item()


# several rounds of CTAs: tiles of up to 256 pairs (one an expert), of up to 128 with an expert's pairs dealt to two, to three, and one tile an expert
@pytest.mark.parametrize("T", [1300, 1800, 2600, 500])
@pytest.mark.parametrize("kind", ["silu", "relu2"])
def test_many_tiles(T, kind):
    test_prompt_experts(T, 136, 1024, 32, 4, kind)


def test_negative_ids_name_no_expert():
    """as those at or beyond the experts: the same bits"""
    from ktransformers_b200.operators.experts import KExpertsDense
    T, width, ff, E, top = 70, 256, 136, 4, 3
    g = torch.Generator(device="cuda").manual_seed(7)
    op = KExpertsDense(width, ff, E)
    for p in (op.gate, op.up, op.down):
        p.data.copy_(torch.randn(p.shape, generator=g, device="cuda") * 0.1)
    x, w = torch.randn((T, width), generator=g, device="cuda").to(torch.bfloat16), torch.rand((T, top), generator=g, device="cuda") + 0.5
    ids = torch.stack([torch.randperm(E, generator=g, device="cuda")[:top] for _ in range(T)])
    ids[::3, 1] = E + 9
    ids[5] = E
    want = op.forward_grouped(x, ids, w)
    assert (want[5] == 0).all()
    assert torch.equal(op.forward_grouped(x, torch.where(ids >= E, E - 1 - ids, ids), w), want)      # -1 and -10
