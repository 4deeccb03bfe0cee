"""A kernel choice that another build saved (OCS_TUNE_CACHE) does not decide:
its lines name no kernel set, or another one, and the request is timed again."""
import os
import re
import shutil
import subprocess

import pytest

from tests.test_api_fake_cuda import _build, _env


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if not shutil.which(os.environ.get("CXX", "g++")):
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("tune_cache") / "api_stress")
    r = _build(out, [])
    assert r.returncode == 0, r.stderr[-4000:]
    return out


def _run(exe, mode, cache):
    return subprocess.run([exe, mode, str(cache)], capture_output=True, text=True, timeout=300, env=_env())


@pytest.mark.parametrize("variant", [r"\2", r"k1:\2", r"k999:\2"])
def test_other_builds_choices_are_timed_again(exe, tmp_path, variant):
    cache = tmp_path / "tune.txt"
    assert _run(exe, "tune-cache-write", cache).returncode == 0
    own = cache.read_text()
    assert _run(exe, "tune-cache-read", cache).returncode == 0
    other = re.sub(r"\|(k\d+:)?(\d+)$", "|" + variant, own, flags=re.M)
    assert other != own or variant == r"\2"
    cache.write_text(other)
    # the request has to time the variants, and no event can be created here
    r = _run(exe, "tune-cache-read", cache)
    assert r.returncode != 0 and "kernel variant timing" in r.stdout, r.stdout + r.stderr
