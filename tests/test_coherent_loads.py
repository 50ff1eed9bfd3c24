"""Kernels that launch_chained starts are alive while the launch before them still
writes, so what that launch writes (links, generator words, counters) may not be read
by the non-coherent path, which asks for data that nothing writes meanwhile.  Read off
the sources: the headers those kernels are made of name no such load, and the batch
names it for its tables alone, which are written when the batch is created."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "qcd_2d_gpu_b200", "csrc")
NON_COHERENT = re.compile(r"\b__ldg\s*\(([^()]*)|ld\.global(?:\.\w+)*\.nc\b")


def code(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"/\*.*?\*/|//[^\n]*", "", src, flags=re.S)


@pytest.mark.parametrize("name", ["lattice.cuh", "sites.cuh", "updates.cuh", "paired.cuh", "kernels.cuh",
                                  "resident.cuh"])
def test_stores_of_chained_kernels_read_coherently(name):
    assert not NON_COHERENT.findall(code(name))


def test_batch_reads_only_its_tables_otherwise():
    found = [m.group(0) for m in NON_COHERENT.finditer(code("batch.cu"))]
    assert found and all("cta_rep" in f for f in found), found
