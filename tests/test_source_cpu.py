"""Rules of the kernels' source that no run shows reliably: they are checked on the text of csrc/."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "benchmark_spmv_using_csr_gb300", "csrc")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            yield name, re.sub(r"//[^\n]*", "", f.read())


def test_carry_records_are_not_read_as_constant_data():
    """The kernels that add the carry records begin while the tile kernel still writes them: a const
    __restrict__ pointer to them would permit the non-coherent load and a load ahead of the wait."""
    for name, text in _sources():
        found = re.findall(r"const\s[^;,(){}]*__restrict__\s+rec_(?:row|val)\b", text)
        assert not found, (name, found)


def test_kernels_raise_errors_at_system_scope():
    """A handle's error word is host memory: kernels set its bits through raise_error, which is atomic
    for the CPU too."""
    for name, text in _sources():
        assert not re.findall(r"\batomicOr\(\s*(?:a\.)?err\b", text), name
    common = dict(_sources())["common.cuh"]
    assert re.search(r"void raise_error\([^)]*\) \{ atomicOr_system\(", common)
