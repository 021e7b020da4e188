"""A head's tokens chosen in its product, where many logits of a row are so close that the order of the sums decides: the
tokens that ``sample`` chooses from the logits of the same head."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _near_ties(rows, vocab, k):
    """Every row's halves along K are the same numbers, and a column has at each place of the first half one of two numbers
    and at that place of the second half the other: equal sums, each rounded by the order it is taken in."""
    g = torch.Generator().manual_seed(rows + vocab + k)
    a = torch.randn(rows, k // 2, generator=g).repeat(1, 2)
    pair = torch.randn(2, k // 2, generator=g)
    pick = torch.randint(0, 2, (vocab, k // 2), generator=g).bool()
    w = torch.cat([torch.where(pick, pair[0], pair[1]), torch.where(pick, pair[1], pair[0])], 1)
    return a.to(DEV), w.bfloat16().to(DEV).contiguous(), torch.randn(vocab, generator=g).mul_(1e-6).to(DEV)


# ring-fed: one row to sixteen, fewer columns than SMs and a group of eight with a remainder, one piece of K and several
# (768, 1088, 2112, 4160); bulk-fed and register-fed; 17 to 64 rows narrow with a long K, tiles that a product that is no head cuts
# along K (9500 x 4096, 5003 x 4096 of 100 rows)
@pytest.mark.parametrize("rows,vocab,k", [
    (8, 32000, 768), (3, 512, 64), (1, 2, 64), (16, 5004, 1600), (9, 1190, 1088), (2, 4738, 2112), (5, 200, 4160), (16, 9470, 1024),
    (8, 50256, 768), (12, 30011, 1600), (32, 4096, 4096), (20, 5003, 2048), (40, 9500, 4096), (100, 5003, 4096), (150, 20011, 136)])
def test_tokens_are_those_of_the_heads_logits(rows, vocab, k):
    a, w, b = _near_ties(rows, vocab, k)
    a = a.bfloat16()
    # rows of logits an even and an odd number of elements apart
    for bias, pad in ((None, 0), (b, 1)):
        logits = torch.empty(rows, vocab + pad, device=DEV)[:, :vocab]
        K.linear(a, w, bias, logits, head=True)
        exact = a.double() @ w.double().T + (0.0 if bias is None else bias.double())
        assert (logits.double() - exact).abs().max().item() <= 8 * k * 2.0 ** -24 * max(1.0, exact.abs().max().item())
        logits = logits.contiguous()
        if not K.sampling_product_possible(rows, vocab, k, torch.bfloat16):
            continue
        want, got = (torch.empty(rows, dtype=torch.int32, device=DEV) for _ in range(2))
        K.sample(logits, None, None, None, None, None, want)
        for _ in range(2):  # its scratch is left zero
            got.fill_(-7)
            K.linear_sample(a, w, bias, K.SampleInto(got))
            assert torch.equal(got, want)
        temps = torch.tensor([0.7, 0.0, 1.0, 1.3], device=DEV).repeat(40)[:rows].contiguous()
        seeds, counters = torch.arange(rows, device=DEV) * 7919, torch.arange(rows, dtype=torch.int32, device=DEV)
        K.sample(logits, temps, None, None, seeds, counters, want)
        K.linear_sample(a, w, bias, K.SampleInto(got, temps, seeds, counters))
        assert torch.equal(got, want)
    K.check_status(torch.device(DEV))


@pytest.mark.parametrize("rows,vocab,k", [(1, 32000, 768), (8, 1190, 1024), (16, 516, 64)])
def test_tokens_of_normalised_rows_reach_the_host_too(rows, vocab, k):
    x, w, _ = _near_ties(rows, vocab, k)
    gamma = torch.randn(k // 2, device=DEV).repeat(2)
    h = K.NormInput(x, gamma, None, 1e-5)
    logits, want, got = torch.empty(rows, vocab, device=DEV), *(torch.empty(rows, dtype=torch.int32, device=DEV) for _ in range(2))
    ring, step = torch.full((K.SAMPLE_RING, 16), -1, dtype=torch.int32).pin_memory(), torch.zeros(1, dtype=torch.int32, device=DEV)
    into = K.SampleInto(got, host_ring=ring, ring_step=step)
    for cap in (0.0, 5.0):  # (the arg-max is the same with and without a bound)
        K.linear(h, w, None, logits, head=True)
        K.sample(logits, None, None, None, None, None, want)
        K.linear_sample(h, w, None, into, soft_cap=cap)
        torch.cuda.synchronize()
        assert torch.equal(got, want) and ring[int(step) - 1, :rows].tolist() == want.tolist()
    assert int(step) == 2
    K.check_status(torch.device(DEV))


def test_rows_that_are_not_numbers_choose_as_the_sampling_kernel_does():
    a = torch.randn(3, 768, device=DEV).bfloat16()
    w = torch.randn(1000, 768, device=DEV).bfloat16()
    w[::3] = float("nan")
    w[1::3, 0], a[1, 0] = float("inf"), -1.0  # -inf in two thirds of the other entries
    a[0, 0] = 0.5
    logits, want, got = torch.empty(3, 1000, device=DEV), *(torch.empty(3, dtype=torch.int32, device=DEV) for _ in range(2))
    K.linear(a, w, None, logits, head=True)
    K.sample(logits, None, None, None, None, None, want)
    K.linear_sample(a, w, None, K.SampleInto(got))
    assert torch.equal(got, want)
