"""The flash kernels (head size 64) at the edges of their 64- and 128-row blocks, against float64 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# P, dS and every result are rounded to 8 bits (2^-9 relative at most each); two full roundings bound the 2-norm, and twice
# that the gradients, whose products carry the rounding of dS as well
BF16_REL = 2 * 2.0 ** -8


def _reference(q, k, v, do, causal):
    leaves = [t.double().requires_grad_(True) for t in (q, k, v)]
    s = leaves[0] @ leaves[1].transpose(1, 2) / 8
    if causal:
        s = s.masked_fill(torch.ones(s.shape[1:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    out = torch.softmax(s, -1) @ leaves[2]
    return out.detach(), torch.logsumexp(s, -1).detach(), torch.autograd.grad(out, leaves, do.double())


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("T", [1, 63, 64, 65, 127, 128, 129, 191, 192, 193, 257, 520])
def test_every_remainder_of_a_block(T, causal):
    from cme213_final_project_b200 import ops
    H = 5
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v, do = (torch.randn(T, H * 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    out, lse = ops.attention_fwd(q, k, v, 1, H, T, "split", causal, backend="tc")
    runs = {m: ops.attention_bwd(q, k, v, out, lse, do, 1, H, T, "split", causal, backend="tc", dq_mode=m) for m in (0, 1)}
    assert ops.attention_check_status() == 0
    heads = [t.reshape(T, H, 64).transpose(0, 1) for t in (q, k, v, do)]
    ref, ref_lse, ref_grads = _reference(*heads, causal)
    back = lambda t: t.transpose(0, 1).reshape(T, H * 64)                    # noqa: E731
    assert ((out.double() - back(ref)).norm() / ref.norm()).item() < BF16_REL
    assert (lse.double() - ref_lse.reshape(-1)).abs().max().item() < 1e-4
    for grads in runs.values():
        for got, want in zip(grads, ref_grads):
            err = (got.double() - back(want)).norm().item()
            # one visible key: dS = P (dP - delta) cancels to rounding noise, compare with dO's size
            assert err < (2 * BF16_REL * want.norm().item() if T > 1 else 2.0 ** -4)


@pytest.mark.parametrize("T,causal", [(256, True), (520, False), (1024, True)])
def test_the_same_call_gives_the_same_bits(T, causal):
    """Scores are written over the probabilities of the block before: were they not held back until the products that read those
    are complete, which bits come out would depend on what else the SM runs.  (dQ is added up in arrival order.)"""
    from cme213_final_project_b200 import ops
    B, H = 16, 12
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v, do = (torch.randn(B * T, H * 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    runs = []
    for _ in range(8):
        out, lse = ops.attention_fwd(q, k, v, B, H, T, "split", causal, backend="tc")
        _, dk, dv = ops.attention_bwd(q, k, v, out, lse, do, B, H, T, "split", causal, backend="tc")
        runs.append((out, lse, dk, dv))
    assert ops.attention_check_status() == 0
    for run in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(run, runs[0]))


def _many(T):
    """Heads enough for the small CTAs in both directions (a few take the kernels with 128 x 128 blocks)."""
    return 900 // -(-T // 128) + 1


def _wide(heads, T, causal, backward):
    from cme213_final_project_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return bool(ops.lib().cme_attention_tc_wide(heads, T, int(causal), int(backward), sms))


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("T", [1, 63, 64, 65, 127, 128, 129, 191, 192, 193, 257, 520])
def test_small_and_wide_kernels(T, causal):
    """The same heads in a call of a few (128 x 128 blocks) and in one of many (64 x 128): both against float64, and every copy of a
    head gets the same bits."""
    from cme213_final_project_b200 import ops
    H = 5
    copies = _many(T) // H + 1
    assert all(_wide(H, T, causal, b) and not _wide(H * copies, T, causal, b) for b in (False, True))
    g = torch.Generator(device="cuda").manual_seed(T)
    few = [torch.randn(T, H * 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4)]
    ref, ref_lse, ref_grads = _reference(*(t.reshape(T, H, 64).transpose(0, 1) for t in few), causal)
    back = lambda t: t.transpose(0, 1).reshape(T, H * 64)                    # noqa: E731
    for n in (1, copies):
        q, k, v, do = (t.repeat(n, 1) for t in few)
        out, lse = ops.attention_fwd(q, k, v, n, H, T, "split", causal, backend="tc")
        dq, dk, dv = ops.attention_bwd(q, k, v, out, lse, do, n, H, T, "split", causal, backend="tc")
        assert ops.attention_check_status() == 0
        for t in (out, dk, dv, lse):                        # (dQ is added up in arrival order)
            t = t.view(n, -1)
            assert (t == t[:1]).all()
        assert ((out[:T].double() - back(ref)).norm() / ref.norm()).item() < BF16_REL
        assert (lse[:H * T].double() - ref_lse.reshape(-1)).abs().max().item() < 1e-4
        for got, want in zip((dq, dk, dv), ref_grads):
            for i in {0, n - 1}:
                err = (got[i * T:(i + 1) * T].double() - back(want)).norm().item()
                # one visible key: dS = P (dP - delta) cancels to rounding noise, compare with dO's size
                assert err < (2 * BF16_REL * want.norm().item() if T > 1 else 2.0 ** -4)


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("T", [65, 96, 130, 200, 256])
def test_a_key_that_an_infinite_element_hides(T, causal, many):
    """Every score of the key is -inf, so it gets no weight and no gradient; the rows of the last block beyond T are zeros, and
    0 x inf must not reach the gradients either."""
    from cme213_final_project_b200 import ops
    H, j = _many(T) if many else 3, T // 2
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v, do = (torch.randn(T, H, 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    q[:, :, 3] = q[:, :, 3].abs() + 0.5
    k[j, :, 3] = float("-inf")
    flat = [t.reshape(T, H * 64) for t in (q, k, v, do)]
    out, lse = ops.attention_fwd(*flat[:3], 1, H, T, "split", causal, backend="tc")
    ref, ref_lse, ref_grads = _reference(*(t.transpose(0, 1) for t in (q, k, v, do)), causal)
    rel = lambda a, b: ((a.double().reshape(T, H, 64).transpose(0, 1) - b).norm() / b.norm()).item()          # noqa: E731
    assert rel(out, ref) < BF16_REL and (lse.double() - ref_lse.reshape(-1)).abs().max().item() < 1e-4
    seen = torch.arange(64, device="cuda") != 3             # dQ = dS K is NaN in the element's column, as it has to be
    for mode in (0, 1, 2):
        dq, dk, dv = ops.attention_bwd(*flat[:3], out, lse, flat[3], 1, H, T, "split", causal, backend="tc", dq_mode=mode)
        assert rel(dk, ref_grads[1]) < 2 * BF16_REL and rel(dv, ref_grads[2]) < 2 * BF16_REL
        dq = dq.double().reshape(T, H, 64).transpose(0, 1)[..., seen]
        assert ((dq - ref_grads[0][..., seen]).norm() / ref_grads[0][..., seen].norm()).item() < 2 * BF16_REL
        assert dv.reshape(T, H, 64)[j].abs().max().item() == 0 and dk.reshape(T, H, 64)[j].abs().max().item() == 0


@pytest.mark.parametrize("H", [3, 900])
def test_probability_of_the_largest_of_128_keys_is_exact(H):
    """The second block of 64 keys holds a row's largest score, less than the rescaling threshold above the first block's: the
    probability is 1 at the reference maximum only, and anything else is rounded to 8 bits before it is multiplied with V."""
    from cme213_final_project_b200 import ops
    T = 128
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k = (torch.zeros(T, H, 64, device="cuda") for _ in range(2))
    v = torch.randn(T, H, 64, generator=g, device="cuda")
    q[..., 0] = 3 + 2.3 * torch.rand(T, H, generator=g, device="cuda")       # scores 3 to 5.3, log2 4.3 to 7.6, of key 100,
    k[..., 0], k[5, :, 0], k[100, :, 0] = -64, 0, 8                          # 0 of key 5, -24 and less of the others
    q, k, v = (t.to(torch.bfloat16).reshape(T, H * 64) for t in (q, k, v))
    out, _ = ops.attention_fwd(q, k, v, 1, H, T, "split", False, backend="tc")
    heads = [t.reshape(T, H, 64).transpose(0, 1) for t in (q, k, v)]
    ref, _, _ = _reference(*heads, torch.zeros_like(heads[0]), False)
    rounding = ((ref.to(torch.bfloat16).double() - ref).norm() / ref.norm()).item()
    err = ((out.reshape(T, H, 64).transpose(0, 1).double() - ref).norm() / ref.norm()).item()
    # the result is rounded, and the probability of key 5 (a weight of 5 % at most); rounding that of key 100 too gives 1.4
    assert err < 1.1 * rounding
