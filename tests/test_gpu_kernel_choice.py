"""Which kernel a request runs: the default of every window, and what OCS_KERNEL
makes of it.  An OCS_KERNEL that does not apply to a window is a preference, so a
test that forces a kernel covers only the windows where this table names it."""
import pytest

pytestmark = pytest.mark.gpu
ONE, PAIR, LANES, MIRROR = 0, 2, 3, 4  # ocs_plan_tune's variants
HALF = "--half_complex_return"


def default(exp, half):
    if exp >= 12:
        return MIRROR
    if half:
        return LANES if exp == 6 else ONE
    return LANES if exp <= 8 else PAIR if exp <= 10 else ONE


def forced(kernel, exp, half):
    if kernel == "single":
        return ONE
    if kernel == "pair":
        if exp in (6, 8, 9, 10):
            return PAIR
        return ONE if exp >= 12 else default(exp, half)
    if kernel == "tpf" and (exp == 6 or (exp <= 8 and not half)):
        return LANES
    if kernel == "x2" and exp >= 12:
        return MIRROR
    return default(exp, half)


@pytest.mark.parametrize("kernel", ["", "single", "pair", "tpf", "x2"])
@pytest.mark.parametrize("opts", ["", "--serial_power", "--layout=dense", HALF, HALF + " --layout=dense"])
@pytest.mark.parametrize("exp", list(range(6, 16)))
def test_variant_of_every_window(ocs_lib, monkeypatch, exp, opts, kernel):
    monkeypatch.setenv("OCS_AUTOTUNE", "0")
    monkeypatch.setenv("OCS_KERNEL", kernel)
    assert ocs_lib.plan_tune(5 << exp, exp, 0.5, opts) == forced(kernel, exp, HALF in opts)


@pytest.mark.parametrize("opts", ["", "--serial_power", HALF, HALF + " --layout=dense"])
@pytest.mark.parametrize("exp", list(range(6, 16)))
def test_tuner_keeps_the_accuracy(ocs_lib, exp, opts):
    """The tuner's own pick never puts two frames in one FFT where that is not
    the window's rule, nor the two-level twiddles beside a one-frame mirror."""
    half = HALF in opts
    pair_ok = exp in (6, 10) if half else exp in (6, 9, 10, 12, 13)
    for n in (1 << 17, 1 << 21, 1 << 24):
        v = ocs_lib.plan_tune(n, exp, 0.5, opts)
        two = v == PAIR or (v == MIRROR and exp <= 13 and not half)
        assert pair_ok or not two, (n, v)
        if exp >= 14 or (exp == 13 and half):
            assert v == MIRROR, (n, v)
