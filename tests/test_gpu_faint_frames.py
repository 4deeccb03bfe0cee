"""A quiet frame beside a loud one.  Kernels that hold one frame per FFT give every
frame its own accuracy; two frames in one FFT round relative to the louder.  The
windows and outputs below hold one frame per FFT, in the one-request entry with
and without the tuner and in batches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
POWER, SERIAL, HALF = "", "--serial_power", "--half_complex_return"
DENSE = " --layout=dense"
ONE_REQUEST = [(e, POWER) for e in (6, 7, 8, 11, 14, 15)] + [(8, SERIAL)] + [(e, HALF) for e in (6, 7, 8, 9, 11, 12, 13, 14, 15)]
BATCH = ([(e, POWER) for e in (6, 7, 8, 11, 13)] + [(e, SERIAL) for e in range(6, 14)] +
         [(e, HALF) for e in range(6, 14)])


def _frames(exp, frames):
    """Frames in the pattern loud, quiet, quiet, loud, .., and at the end silence beside a loud one."""
    N = 1 << exp
    level = np.where(np.arange(frames) % 4 % 3 == 0, 1.0, 1e-4)
    level[-2:] = 0.0, 1.0
    x = np.random.default_rng(exp).uniform(-1, 1, (frames, N)) * level[:, None]
    return x.astype(np.float32)


def _check(got, x, opts):
    frames, N = x.shape
    half = HALF in opts
    row = N // 2 + 1 if DENSE in opts else N
    want = np.fft.fft(x.astype(np.float64))[:, :row]
    if not half:
        want = np.sqrt(2) * np.abs(want.real) if SERIAL in opts else np.abs(want)
    got = got.astype(np.float64)
    if half:
        got = got.view(np.complex128)
    n = min(frames, got.size // row)  # the reference's half-complex layout holds half of the frames
    got = got[:n * row].reshape(n, row)
    for f in range(n):
        # the repository's bar for spectra, frame by frame
        assert np.linalg.norm(got[f] - want[f]) <= 1e-5 * np.linalg.norm(want[f]), (f, opts)


def _run(ocs, x, exp, opts, batch):
    import torch

    d = torch.from_numpy(x.reshape(-1)).cuda()
    g = ocs.geometry(x.size, exp, 0.0, opts)
    out = torch.zeros(g.out_floats, device="cuda")
    if batch:
        assert ocs.batch_device(ocs.make_requests([(d, x.size, exp, 0.0, opts, out, g.out_floats)])) == [0]
    else:
        ocs.activate_device(d, x.size, exp, 0.0, opts, out, g.out_floats)
    return out.cpu().numpy()


@pytest.mark.parametrize("tune", ["0", "1"])
@pytest.mark.parametrize("layout", ["", DENSE])
@pytest.mark.parametrize("exp,opts", ONE_REQUEST)
def test_one_request(ocs_lib, monkeypatch, exp, opts, layout, tune):
    monkeypatch.setenv("OCS_AUTOTUNE", tune)
    # a few frames, and enough for the tuner to see the kernels' own speeds; at 2^6
    # it may take two frames per FFT for a few
    for frames in (8, max(8, (1 << 22) >> exp)):
        if exp == 6 and tune == "1" and frames == 8:
            continue
        x = _frames(exp, frames)
        _check(_run(ocs_lib, x, exp, opts + layout, False), x, opts + layout)


@pytest.mark.parametrize("layout", ["", DENSE])
@pytest.mark.parametrize("exp,opts", BATCH)
def test_batch(ocs_lib, exp, opts, layout):
    for frames in (8, max(8, (1 << 20) >> exp)):
        x = _frames(exp, frames)
        _check(_run(ocs_lib, x, exp, opts + layout, True), x, opts + layout)
