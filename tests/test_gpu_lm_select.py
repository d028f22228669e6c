"""The C best logits of the LM head: vocabularies around a slice of 256, slices longer than that, and more equal logits than
the collecting buffer holds."""
import pytest

torch = pytest.importorskip("torch")
import rlx_b200 as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_vocab,cap,equal", [(9, 9, False), (255, 3, False), (257, 64, False), (5000, 64, False), (524289, 40, False),
                                               (600000, 1, False), (20000, 40, True), (700000, 64, True)])
def test_selection_is_the_sorted_logits(n_vocab, cap, equal):
    g = torch.Generator(device="cuda")
    g.manual_seed(n_vocab)
    k, scheme = 64, R.QuantScheme.GgufQ4_0
    w = torch.randint(0, 256, (n_vocab * k // 32, 18), dtype=torch.uint8, device="cuda", generator=g)
    w[:, :2] = torch.full((1,), 0.01, device="cuda").half().view(torch.uint8)
    w = w.reshape(-1)
    x = torch.zeros((1, k), device="cuda") if equal else torch.randn((1, k), device="cuda", generator=g)
    logits = R.matmul(x, w, scheme, n_vocab)[0]
    val, idx = torch.sort(logits, descending=True, stable=True)
    got_i, got_v = R.gguf_tied_lm_topk(x[0].contiguous(), w, k, n_vocab, scheme, cap, exact=False)
    assert torch.equal(got_i.long(), idx[:cap])
    assert torch.equal(got_v, val[:cap])
