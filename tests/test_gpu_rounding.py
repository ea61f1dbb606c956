"""Records before the wave's arrival, which are the transforms' rounding, are
those of the earlier library, bit for bit (tests/golden/make_rounding.py says
why): the same products are rounded in the same order, whatever form a kernel
has."""
import importlib.util
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

spec = importlib.util.spec_from_file_location("make_rounding", os.path.join(GOLDEN, "make_rounding.py"))
mk = importlib.util.module_from_spec(spec)
spec.loader.exec_module(mk)


@pytest.fixture(scope="module")
def kept():
    return np.load(os.path.join(GOLDEN, "rounding", "records.npz"))


@pytest.mark.parametrize("name", sorted({**mk.SHOTS, **mk.TC}))
def test_records(qvti, kept, name):
    assert np.array_equal(mk.shot(qvti, name), kept[name])


@pytest.mark.parametrize("name", sorted(mk.RTM))
def test_images(qvti, kept, name):
    assert np.array_equal(mk.rtm(qvti, name), kept[name])
