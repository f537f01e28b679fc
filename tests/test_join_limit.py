"""Joined fronts stay within the rows that a solve's shared memory holds.

The symbolic analysis alone, on the CPU: joins of a 40 x 40 grid's levels with
no limit that matters, with one between the largest front of the dissection
and the largest joined one, and without joins.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    csrc = os.path.join(os.path.dirname(HERE), "doug_gb300", "csrc")
    exe = str(tmp_path_factory.mktemp("join") / "join_limit")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", csrc, os.path.join(HERE, "join_limit.cpp"),
                    os.path.join(csrc, "host", "mf_symbolic.cpp"), "-o", exe], check=True)
    return lambda limit, thin: tuple(map(int, subprocess.run([exe, "40", str(limit), str(thin)], capture_output=True,
                                                             text=True, check=True).stdout.split()))


def test_joined_fronts_are_limited(program):
    joined, levels = program(0, 100000)
    plain, plain_levels = program(0, 0)
    assert levels < plain_levels and joined > plain
    limit = (joined + plain) // 2
    some, some_levels = program(limit, 100000)
    assert some <= limit
    assert levels < some_levels < plain_levels
