"""Operand copies and gradient export of all members at once, against the linears' own methods."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BUFFERS = ("A_cat", "A_catT", "B_cat", "B_catT")


# ranks below, at and above a group of 8 and a pass of 32; sizes off the 64-wide tiles; a member that has no adapter
@pytest.mark.parametrize("r,K,n", [(1, 64, 16), (8, 200, 48), (12, 72, 80), (40, 328, 144)])
def test_all_members_at_once(r, K, n):
    from art_b200.models.native import LoraLinear, _Member
    from art_b200.ops.lora_pack import LoraTable

    g = torch.Generator(device=DEV).manual_seed(r)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    i = torch.arange(n, device=DEV)
    gate = (i // 16) * 32 + i % 16
    lins = []
    for rows in ([gate, gate + 16], [i], [], [torch.arange(n // 2, device=DEV), torch.arange(n // 2, n, device=DEV)]):
        members = [_Member("m", rw, j, rnd(r, K), rnd(rw.numel(), r), rnd(r, K), rnd(rw.numel(), r)) for j, rw in enumerate(rows)]
        lins.append(LoraLinear(rnd(max(n, 2 * n if len(rows) == 2 else n), K).bfloat16(), None, members, r, 1.7))
    act = [lin for lin in lins if lin.active]
    for lin in act:
        lin.refresh()
    want = [{k: getattr(lin, k).clone() for k in BUFFERS} for lin in act]
    for lin in act:
        for k in BUFFERS:
            getattr(lin, k).zero_()
    table = LoraTable(lins)
    table.refresh()
    for lin, w in zip(act, want):
        assert all(torch.equal(getattr(lin, k), w[k]) for k in BUFFERS)
        lin.dA_acc.copy_(rnd(*lin.dA_acc.shape))
        lin.dB_acc.copy_(rnd(*lin.dB_acc.shape))
        lin.export_grads()
    grads = [t for lin in act for m in lin.members for t in (m.ga_view, m.gb_view)]
    ref = [t.clone() for t in grads]
    for t in grads:
        t.zero_()
    table.export_grads()
    assert all(torch.equal(a, b) for a, b in zip(grads, ref))
    table.zero_grad()
    assert all(not bool(t.any()) for lin in act for t in (lin.dA_acc, lin.dB_acc))
