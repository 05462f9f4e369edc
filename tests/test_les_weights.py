"""Weights set from the host reach every packed form of them: the tensor-core gradients and
the inference after set_weights equal those of the network the weights came from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_gradients_after_set_weights(ns3d):
    D = 16
    a, b = ns3d.LES(D, capacity=0, seed=5), ns3d.LES(D, capacity=0, seed=6)
    for les in (a, b):
        les.set_scales(1.2, 0.8)
    b.set_weights(a.weights())
    rng = np.random.default_rng(1)
    u = rng.standard_normal((3, D, D, D)).astype(np.float32)
    t = rng.standard_normal((6, D, D, D)).astype(np.float32) * 0.1
    (la, ga), (lb, gb) = a.gradients(u, t), b.gradients(u, t)
    assert la == lb and np.array_equal(ga, gb)
    assert np.array_equal(a.infer(u), b.infer(u))
    a.close()
    b.close()
