"""The shares of the assembled cluster CG (lpm-cpp_b200/csrc/shares.cuh, on the host).

A CTA of that kernel takes part in an exchange by sending the sums and the residual of its slices, and the
others store into it only after that.  So a CTA without a slice would be waited for by nobody while the
others store into it, and every share must hold one: also where the slices do not divide evenly (58 slices
on 16 CTAs leave the last one empty when each takes four) and where there are fewer slices than CTAs."""
import os
import subprocess

import pytest

from _util import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("limit", [8, 16])
def test_every_cta_has_a_slice(limit, tmp_path):
    exe = str(tmp_path / "shares_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "lpm-cpp_b200", "csrc"),
                    os.path.join(HERE, "native", "shares_check.cpp"), "-o", exe], check=True)
    lines = subprocess.run([exe, "148", str(limit)], check=True, capture_output=True, text=True).stdout.splitlines()
    assert len(lines) == 148
    for line in lines:
        n, nc, most, *at = map(int, line.split())
        assert 1 <= nc <= limit and nc & (nc - 1) == 0 and len(at) == nc + 1
        sizes = [b - a for a, b in zip(at, at[1:])]
        assert at[0] == 0 and at[-1] == n
        assert min(sizes) >= 1 and max(sizes) == most, (n, sizes)
        assert nc == limit or 2 * nc > n
