"""The FP32 triangle test of the contact search, compiled for the host: no contact is lost on triangles of any length and
width, the short edge at each vertex in turn, near the origin and far from it, and spheres clear of an ordinary triangle
are told apart."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("near") / "triangle_near")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(HERE, "..", "metakonga_gb300", "csrc"), "-o", out,
                    os.path.join(HERE, "cpp", "triangle_near.cpp")], check=True)
    return out


@pytest.mark.parametrize("far", [0.0, 0.3, 20.0, 1e4])
def test_no_contact_is_lost(program, far):
    got = subprocess.run([program, "2000", str(far)], check=True, capture_output=True, text=True).stdout
    contacts, lost, clear, called = map(int, got.split())
    assert contacts > 1_000_000 and lost == 0
    if far <= 1.0:
        assert clear > 1_000 and called == 0
