"""The PSF's row-spectrum chunk as the environment sets it (host queries only;
the library reads its settings once, so each is tried in its own process)."""

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

QUERY = """
from chromatix_b200 import _native as nat
d = nat.cx_psf_desc()
d.ny, d.nx, d.n_wv, d.n_z, d.f_lens = 1280, 1280, 3, 64, 1.0
b = nat.c_size_t(0)
nat.check(nat.lib().cx_psf_workspace_size(d, b))
print(b.value)
"""


def _workspace(**env):
    e = {k: v for k, v in os.environ.items() if not k.startswith("CX_PSF_")}
    e.update(env)
    out = subprocess.run([sys.executable, "-c", QUERY], cwd=ROOT, env=e, capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    return int(out.stdout)


@pytest.fixture(scope="module")
def default():
    return _workspace()


@pytest.mark.parametrize("name", ["CX_PSF_CHUNK_MB", "CX_PSF_L2_MB"])
@pytest.mark.parametrize("mb", [64, 100])
def test_chunk_in_mib(default, name, mb):
    # default: 512 MiB of row spectra; the rest of the workspace does not depend on the chunk
    assert default - _workspace(**{name: str(mb)}) == (512 - mb) << 20


def test_the_newer_name_decides(default):
    assert default - _workspace(CX_PSF_CHUNK_MB="100", CX_PSF_L2_MB="64") == (512 - 100) << 20


@pytest.mark.parametrize("value", ["0", "-5", "many", ""])
def test_no_number_is_the_default(default, value):
    assert _workspace(CX_PSF_CHUNK_MB=value) == default
    assert _workspace(CX_PSF_L2_MB=value) == default
