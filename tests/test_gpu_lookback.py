"""A look-back whose bounded wait runs out must end as an error of the call, not
as an index into some array: the scans and the sort are built with a switch that
makes chosen ones give up, linked with the library's other objects."""
import os
import subprocess
import sys

import pytest

from pike_gb300 import build as pk_build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_builders_report_a_look_back_that_gave_up(pk_built, tmp_path):
    pytest.importorskip("torch")
    objs = [os.path.join(pk_build.BUILD_DIR, s.rsplit(".", 1)[0] + ".o") for s in pk_build.SOURCES]
    if not all(os.path.exists(o) for o in objs):
        pk_build.build(force=True)
    util, lib = str(tmp_path / "pk_util.o"), str(tmp_path / "libpike_gives_up.so")
    cc = pk_build.nvcc()
    subprocess.run([cc, *pk_build.ARCH, *pk_build.NVFLAGS, "-include", os.path.join(HERE, "lookback_gives_up.cuh"), "-c",
                    os.path.join(pk_build.CSRC, "pk_util.cu"), "-o", util], check=True)
    subprocess.run([cc, *pk_build.ARCH, "-shared", "-o", lib, util,
                    *[o for o in objs if not o.endswith("pk_util.o")], "-lpthread"], check=True)
    r = subprocess.run([sys.executable, os.path.join(HERE, "lookback_child.py"), lib], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr
