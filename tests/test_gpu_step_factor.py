"""The step factor 0.9 / maxerr^(1/3) of an accepted ROS3 step (csrc/ros3.cuh) on the device against
extended precision, for every size of error norm that a step can be accepted with."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CLIP = (0.9 / 10.0) ** 3      # below it the factor is clipped at FACMAX = 10


def test_step_factor():
    from cmaq_gb300 import _lib
    rng = np.random.default_rng(11)
    n = 400000
    x = np.concatenate([np.exp(rng.uniform(np.log(CLIP), 0.0, n)), 1.0 - rng.random(n) * (1.0 - CLIP),
                        1.0 - np.exp(rng.uniform(np.log(2.0**-53), np.log(0.5), n)),
                        CLIP * (1.0 + np.arange(-n // 4, n // 4) * 2.0**-50),
                        *[2.0**-k * (1.0 + np.arange(0, 1000) * 2.0**-52) for k in range(1, 11)], [1.0]])
    x = x[(x > 0.0) & (x <= 1.0)]
    refined, by_pow = _lib.step_factor(x)
    exact = np.longdouble(0.9) / np.cbrt(x.astype(np.longdouble))
    err = [np.max(np.abs(v - exact) / exact) for v in (refined, by_pow)]
    worst = np.max(np.abs(refined - exact) / np.spacing(exact.astype(np.float64)))
    print(f"refined {float(err[0]):.3g} ({float(worst):.2f} ulp), by pow {float(err[1]):.3g} "
          f"({float(np.max(np.abs(by_pow - exact) / np.spacing(exact.astype(np.float64)))):.2f} ulp)")
    # 2.7 roundings and 4.7 times the third power of the float estimate's error of 1e-6
    assert err[0] <= 2.7 * 2.0**-53 + 4.7e-18
    assert err[0] <= err[1]
    # the largest error norms whose factor is clipped: clipped all the same
    small = np.concatenate([np.exp(rng.uniform(np.log(2.3e-16), np.log(CLIP * (1.0 - 1e-12)), n)), [2.3e-16]])
    assert np.all(_lib.step_factor(small)[0] >= 10.0)
