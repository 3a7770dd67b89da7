"""Router top-k: expert counts on both sides of the register / shared-memory split, ties, and
logits that are not numbers (which must never yield an index outside the experts)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,E,K", [(1, 1, 1), (3, 8, 8), (37, 33, 5), (130, 256, 8), (65, 257, 8), (9, 1000, 32), (5, 12800, 3)])
def test_topk_matches_stable_sort(S, E, K):
    from moonep_b200.ops import elementwise as ew
    g = torch.Generator(device="cuda").manual_seed(E)
    logits = (torch.randn(S, E, device="cuda", generator=g) * 4).round() / 4        # many ties
    bias = (torch.randn(E, device="cuda", generator=g) * 2).round() / 4
    topk, w, tpe = ew.router_topk(logits, K, bias)
    want = torch.sort(logits + bias, dim=1, descending=True, stable=True).indices[:, :K]
    assert torch.equal(topk.long(), want)
    torch.testing.assert_close(w, torch.softmax(logits.gather(1, want), 1), rtol=1e-5, atol=1e-6)
    assert torch.equal(tpe.long(), torch.bincount(want.flatten(), minlength=E))


@pytest.mark.parametrize("E", [48, 300])
def test_not_a_number_and_infinities(E):
    from moonep_b200.ops import elementwise as ew
    K = 4
    logits = torch.zeros(4, E, device="cuda")
    logits[0] = float("nan")
    logits[1] = float("-inf")
    logits[2, ::2] = float("nan")
    logits[2, 7] = 1.0
    logits[3, 5] = float("inf")
    topk, _, tpe = ew.router_topk(logits, K)
    assert topk.cpu().tolist() == [[0, 1, 2, 3], [0, 1, 2, 3], [7, 1, 3, 5], [5, 0, 1, 2]]
    assert int(tpe.sum()) == 4 * K


@pytest.mark.parametrize("E", [40, 300])
def test_zeros_of_either_sign_tie(E):
    """A bias of -0.0 (no popularity at all) beside logits of -0.0: equal values go by the expert's index."""
    from moonep_b200.ops import elementwise as ew
    logits = torch.zeros(3, E, device="cuda")
    logits[0, ::2] = -0.0
    logits[1] = -0.0
    logits[2, 3] = -1.0
    topk, _, _ = ew.router_topk(logits, 4, -torch.zeros(E, device="cuda"))
    assert topk.cpu().tolist() == [[0, 1, 2, 3], [0, 1, 2, 3], [0, 1, 2, 4]]
