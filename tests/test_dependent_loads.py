"""A kernel that starts before the one ahead of it in the stream has ended (programmatic dependent launch)
must not read what that one writes through the read-only path (__ldg, or const __restrict__ pointers, which
the compiler may turn into it), nor by any load that is not kept behind the wait; plain loads are.  Wrong results from that depend on timing, so the sources are read."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "bit-graphblas_gb300" / "csrc"


def function(source, name):
    """Parameters and body, without comments, of the namespace-level function `name`."""
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    m = re.search(rf"\b{name}\(([^;{{}}]*)\)\s*\{{.*?^\}}", text, re.M | re.S)
    assert m, f"{name} is not defined in {source}"
    return m.group(0)


@pytest.mark.parametrize("source,names", [
    ("b2sr_rowbin.cu", ("fixup_group", "rowbin_fixup_kernel", "bits_fixup_group", "rowbin_bits_fixup_kernel")),
    ("b2sr_spmm_rows.cu", ("rows_fixup_kernel",)),
])
def test_slots_are_not_read_only(source, names):
    for name in names:
        body = function(source, name)
        assert not re.search(r"__restrict__\s+partials", body), name
        for line in body.splitlines():
            if re.search(r"__ldc?[agsv]\(|\basm\b", line):  # the plan and the mask: written long before
                assert re.search(r"__ldg\((long_rows|a\.long_rows|static_cast<const W\*>\(a\.mask\))", line), (name, line)
            if "rows_load<" in line:
                assert re.search(r"rows_load<V, VEC, FULL, 32, true>", line), (name, line)


def test_every_dependent_kernel_is_looked_at():
    """The kernels launched that way: those above; and kernels that read the launch before them through plain
    pointers held in their argument struct."""
    launched = set()
    for f in sorted(CSRC.glob("*.cu*")):
        launched |= set(re.findall(r"launch_dependent\((\w+)<", f.read_text()))
    plain = {"push_kernel": ("b2sr_push.cu", ["a.items[i]", "a.ctl[0]"]),
             "rowbin_bits_gate_kernel": ("b2sr_rowbin.cu", ["a.push_ctl[0]"]),
             "carry_fixup_kernel": ("b2sr_spmv_impl.cuh", ["carries[c].row", "carries[c2].val"]),
             "spmm_fixup_kernel": ("b2sr_spmm.cu", ["a.carry_rows[c]", "a.carry_vals +"])}
    assert launched == {"rowbin_fixup_kernel", "rowbin_bits_fixup_kernel", "rows_fixup_kernel"} | set(plain)
    for name, (source, reads) in plain.items():
        body = function(source, name)
        assert all(r in body for r in reads) and "__restrict__" not in body.split("{")[0], name
