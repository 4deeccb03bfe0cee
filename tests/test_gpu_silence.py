"""Digital silence costs what any signal costs: the power kernels' second pass,
for squares below the normal range, is not for bins that are zero."""
import statistics

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["", "--layout=dense"])
@pytest.mark.parametrize("exp", [6, 7, 8, 9, 10, 11, 12, 13, 14, 15])
def test_silent_signal_takes_no_longer(ocs_lib, monkeypatch, exp, layout):
    import torch

    monkeypatch.setenv("OCS_AUTOTUNE", "0")
    n = 1 << 24
    g = ocs_lib.geometry(n, exp, 0.75, layout)
    out = torch.zeros(g.out_floats, device="cuda")
    loud = torch.randn(n, generator=torch.Generator(device="cuda").manual_seed(exp), device="cuda")

    def us(x):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            ocs_lib.activate_device(x, n, exp, 0.75, layout, out, g.out_floats)
        b.record()
        b.synchronize()
        return a.elapsed_time(b) * 100

    silent = torch.zeros_like(loud)
    for x in (loud, silent):
        us(x)
    t = [(us(loud), us(silent)) for _ in range(5)]
    assert float(out.abs().max()) == 0.0
    # the second pass took 1.2 to 1.4 times; the mirror-group kernel's guard is 1.06
    assert statistics.median(s for _, s in t) <= 1.12 * statistics.median(v for v, _ in t), t
