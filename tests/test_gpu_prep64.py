"""The chunk preparation at head dims 64 / 64 (tcgen05 kernel behind ``natsl_gdn_chunk_prep_ex``): remainders of a chunk, the
optional outputs, strong decays, and its error against the formulas in float64."""
import pytest
import torch

from tests.helpers import synth_gdn_inputs
from tests.test_gpu_prep import _check, _reference, _run

pytestmark = pytest.mark.gpu
NAMES = ("gcs", "k_rstd", "q_rstd", "w", "u", "P")
PREP = "natsl_gdn_chunk_prep_ex"


@pytest.mark.parametrize("B,T,H,with_q,beta_f32,l2", [(2, 512, 4, True, False, True), (1, 700, 2, True, True, True),
                                                      (1, 64, 1, False, False, True), (2, 200, 3, True, False, False),
                                                      (1, 1, 1, True, False, True), (1, 33, 2, False, True, True)])
def test_prep64_against_the_formulas(B, T, H, with_q, beta_f32, l2):
    q, k, v, g, beta, _ = synth_gdn_inputs(B, T, H, 64, 64, seed=T + H, normalize_qk=l2 is False)
    if beta_f32:
        beta = beta.float()
    ref = _reference(q, k, v, g, beta, use_l2norm=l2)
    got = _run(PREP, q, k, v, g, beta, with_q, use_l2norm=l2)
    for i, n in enumerate(NAMES):
        if with_q or n not in ("q_rstd", "P"):
            _check(got[i], ref[i], n, 2e-5 if i < 3 else 1e-2)
    again = _run(PREP, q, k, v, g, beta, with_q, use_l2norm=l2)
    assert all(torch.equal(x, y) for x, y in zip(got, again))
    # 2-norm: u and w take one rounding of the inverse, one of k (w) and one of the result, 2^-9 / sqrt(3) each at most; the
    # inverse's entries add up with random signs, so the three together stay below 2^-8
    for i in (3, 4):
        err = (got[i].double().cpu() - ref[i]).norm() / ref[i].norm().clamp_min(1e-30)
        assert err < 2 ** -8, (NAMES[i], float(err))


@pytest.mark.parametrize("beta_f32", [False, True])
@pytest.mark.parametrize("T,decay", [(512, 4.0), (512, 1.0), (1000, 0.05), (512, 0.01)])
def test_prep64_rounds_the_diagonal_once(T, decay, beta_f32):
    """The inverse's diagonal is exactly one: its share of u and w, beta v and beta rstd e^gcs k, reaches the output with the
    output's rounding alone, in bf16 as in fp32 beta.  What is off the diagonal takes two more (the inverse's entry, and k or v)."""
    q, k, v, g, beta, _ = synth_gdn_inputs(1, T, 4, 64, 64, seed=T)
    g = g * decay
    if beta_f32:
        beta = torch.rand(beta.shape, generator=torch.Generator().manual_seed(1))
    ref = _reference(q, k, v, g, beta)
    got = _run(PREP, q, k, v, g, beta, True)
    n = -(-T // 64)
    pad = lambda x: torch.nn.functional.pad(x.double(), (0, 0) * (x.dim() - 2) + (0, n * 64 - T))
    ch = lambda x: pad(x).reshape(1, n, 64, 4, -1).transpose(2, 3)             # [B, chunk, head, token, feature]
    kn, b, gc = ch(k) * ch(ref[1][..., None]), ch(beta[..., None]), ch(g[..., None]).cumsum(-2)
    A = torch.tril(b * (kn @ kn.mT) * (gc - gc.mT).clamp(max=0).exp(), -1)
    off = torch.linalg.inv(torch.eye(64, dtype=torch.float64) + A) - torch.eye(64, dtype=torch.float64)
    for i, rhs in ((3, kn * b * gc.exp()), (4, ch(v) * b)):
        one = (ref[i].bfloat16().double() - ref[i]).norm()                     # what storing the exact result loses
        terms = (off.square() @ rhs.square()).sum() / ref[i].square().sum()    # errors of the products, of independent signs
        err = (got[i].double().cpu() - ref[i]).norm()
        # a tenth for the tf32 products of the inverse (2^-11 of an entry) and the spread of the estimate
        assert err < 1.1 * one * (1 + 2 * terms) ** 0.5, (NAMES[i], float(err / one), float(terms))


def test_prep64_strong_decay_and_large_beta():
    q, k, v, g, beta, _ = synth_gdn_inputs(1, 256, 2, 64, 64, seed=11)
    g, beta = g * 6.0, (beta.float() * 2.0).bfloat16()
    ref = _reference(q, k, v, g, beta)
    for i, (got, n) in enumerate(zip(_run(PREP, q, k, v, g, beta, True), NAMES)):
        _check(got, ref[i], n, 2e-5 if i < 3 else 2e-2)
