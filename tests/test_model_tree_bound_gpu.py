"""The learned dispatcher against a Winograd head that predicts the impossible: a tree's time
is bounded by the plain limb product's, so a head below that bound does not win over
the other plans, and one that the bound allows still does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _heads(g, h, log2ms):
    """A model whose heads give the same prediction for every product."""
    w, _ = h.model_params()
    w = np.zeros_like(w)
    w[-g.NPLANS:] = log2ms
    h.model_set_params(w)
    h.model_use(True)


@pytest.mark.parametrize("shape,ms,plan", [
    # plan 0 (plain), 1 to 3 (trees to 32, 64, 128), 4 to 7 (CRT forms)
    ((93, 50, 37, 5, 4), [0.045, 0.01, 9, 9, 0.022, 0.03, 0.03, 0.04], 4),
    ((160, 160, 160, 3, 3), [0.2, 0.05, 9, 9, 0.14, 0.3, 0.3, 0.3], 4),
    ((160, 160, 160, 3, 3), [0.2, 0.05, 9, 9, 0.19, 0.3, 0.3, 0.3], 1),
])
def test_plan_of_the_model(built_lib, shape, ms, plan):
    import gbmm as g
    m, k, n, la, lb = shape
    h = g.Handle()
    h.model_init(seed=1)
    _heads(g, h, np.log2(np.array(ms, dtype=np.float32)))
    A, B = [(i % 7) - 3 for i in range(m * k)], [(i % 5) - 2 for i in range(k * n)]
    dA, dB = g.DeviceMatrix.from_ints(m, k, A, la), g.DeviceMatrix.from_ints(k, n, B, lb)
    dC = g.DeviceMatrix(m, n, la + lb + 3)
    g.profile(1)
    h.matmul(dC, dA, dB)
    ran = set(g.profile_read())
    g.profile(0)
    if plan >= 4:
        assert any(x.startswith("k_crt") for x in ran), ran
    else:
        assert not any(x.startswith("k_crt") for x in ran), ran
        assert ("k_wino_sums" in ran) == (plan == 1), ran
    exp = np.array(A).reshape(m, k) @ np.array(B).reshape(k, n)
    assert dC.to_ints() == exp.reshape(-1).tolist()
    h.close()
