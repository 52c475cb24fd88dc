"""A look-back whose bounded wait runs out must end as an error of the call, not
as an index into some array: the scans and the sort are built with a switch that
makes chosen ones give up."""
import os

import pytest

from pike_gb300 import build as pk_build

import variant

pytestmark = pytest.mark.gpu


def test_builders_report_a_look_back_that_gave_up(pk_built, tmp_path):
    pytest.importorskip("torch")
    lib = variant.link(str(tmp_path / "libpike_gives_up.so"), [os.path.join(pk_build.CSRC, "pk_util.cu")],
                       ["-include", os.path.join(variant.HERE, "lookback_gives_up.cuh")])
    variant.run("lookback_child.py", lib)
