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


def test_prep64_strong_decay_and_large_beta():
    q, k, v, g, beta, _ = synth_gdn_inputs(1, 256, 2, 64, 64, seed=11)
    g, beta = g * 6.0, (beta.float() * 2.0).bfloat16()
    ref = _reference(q, k, v, g, beta)
    for i, (got, n) in enumerate(zip(_run(PREP, q, k, v, g, beta, True), NAMES)):
        _check(got, ref[i], n, 2e-5 if i < 3 else 2e-2)
