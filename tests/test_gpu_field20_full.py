"""GPU: the 20-source, 8-band x 4-exposure, 128x128 px patch at full size, by
the bars of test_gpu_parity with the float oracle, which restates the reference
CPU kernel operation by operation, in that kernel's place: these run where it
cannot be built."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import CHI2_RTOL, check_grad, gpu_eval, grad_ok

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def field20():
    from forcepho_b200 import synth
    P = synth.make_workload("field20", seed=0)
    prop = P.proposal()
    return (P, prop) + tuple(O.oracle_evaluate(P, prop))


def test_full_size(field20):
    P, prop, c, g = field20
    chi2, dchi2 = gpu_eval(P, prop)
    c64, _ = O.oracle_evaluate(P, prop, precision="f64")
    np.testing.assert_allclose(chi2, c, rtol=CHI2_RTOL)
    np.testing.assert_allclose(chi2, c64, rtol=CHI2_RTOL)
    check_grad(dchi2, g, P, prop)


def test_every_shape(field20):
    """Every compiled tile shape, one CTA per tile and persistent; the second
    persistent evaluation follows the first's costs."""
    from forcepho_b200 import _lib
    from forcepho_b200.proposal import GPUProposer
    P, prop, c, g = field20
    _, mixed, scale, _, rscale = O.oracle_mixed_abs(P, prop, terms=True)
    P.return_residual = False
    P.send_to_device()
    for v in range(len(_lib.variants())):
        for sched in (0, 1):
            P.device_patch.set_config(v, 160)
            P.device_patch.set_schedule(sched)
            for _ in range(2):
                chi2, dchi2 = GPUProposer().evaluate_proposal(prop, patch=P)
            np.testing.assert_allclose(chi2, c, rtol=CHI2_RTOL)
            ok = grad_ok(dchi2, g, mixed, scale, rscale)
            assert np.all(ok), (v, sched, int((~ok).sum()))
    P.free()
