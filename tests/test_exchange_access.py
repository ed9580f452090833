"""The resident sweeps hand edge rows on as {value, step tag} pairs without a
fence, so a pair has to be one access of the memory model.  PTX makes each
element of a vector access a scalar access of its own, in no order: the
exchange's loads and stores have 64-bit elements, a pair each."""
import os
import re

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "swfwi_b200", "csrc")
ACCESS = re.compile(r'"(?:st|ld)\.[\w.]*global[\w.]*')


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_a_pair_is_one_64_bit_access():
    text = source("resident.cuh")
    for name in ("put_pair2", "get_pair2"):
        at = text.index(name + "(")
        accesses = ACCESS.findall(text[at:text.index("\n}\n", at)])
        assert len(accesses) == 1 and accesses[0].endswith(".relaxed.gpu.global.v2.b64"), (name, accesses)


def test_both_sweeps_exchange_by_these_alone():
    assert len(ACCESS.findall(source("resident.cuh"))) == 2
    assert not ACCESS.findall(source("lsrtm_resident.cuh"))
    for name in ("resident.cuh", "lsrtm_resident.cuh"):
        assert "put_pair2(" in source(name) and "get_pair2(" in source(name)
