"""GPU: metadata of another scene that cannot be installed for lack of memory
leave the patch with the scene it had, and the next attempt with enough memory
installs them whole."""
import numpy as np
import pytest

from test_gpu_runs import patch

pytestmark = pytest.mark.gpu

NOMEM = 3


def evaluate(P, scene):
    from forcepho_b200.proposal import GPUProposer
    return GPUProposer().evaluate_proposal(scene.get_proposal(), patch=P, unpack=False)[:2]


def test_replace_meta_without_memory():
    from forcepho_b200 import _lib
    P = patch(12, [1, 1], [(40, 40), (32, 48)], 3, seed=81)
    few, many = P.set_scene(range(2)), P.set_scene(range(12))
    want = {}
    for name, scene in (("few", few), ("many", many)):
        P.pack_meta(scene)
        P.free()
        P.send_to_device()
        want[name] = evaluate(P, scene)
    P.pack_meta(few)
    P.free()
    P.send_to_device()
    P.pack_meta(many)
    failed = 0
    for n in range(1, 20):
        _lib.call("fpho_test_fail_alloc", n)
        try:
            P.replace_device_meta_ptrs()
        except _lib.FphoError as e:
            assert e.code == NOMEM
            failed += 1
        else:
            break
        finally:
            _lib.call("fpho_test_fail_alloc", 0)
        assert P.device_patch.info()["n_sources"] == 2
        P.pack_meta(few)                # the host side of the scene that is installed
        for g, w in zip(evaluate(P, few), want["few"]):
            np.testing.assert_array_equal(g, w)
        P.pack_meta(many)
    assert failed == 5                  # metadata, records, boxes, proposal, partials
    for g, w in zip(evaluate(P, many), want["many"]):
        np.testing.assert_array_equal(g, w)
    P.pack_meta(few)
    P.replace_device_meta_ptrs()        # nothing to allocate
    for g, w in zip(evaluate(P, few), want["few"]):
        np.testing.assert_array_equal(g, w)
    P.free()
