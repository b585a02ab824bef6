"""Faster forms of the device code against the plain ones, built for the host
(tests/arith_host_check.cpp): the polyhedron's hill climb, the divisions by one
reciprocal, the motion test without its square root, the cell index."""
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))


def test_faster_forms_give_the_same_bits():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "arith_host_check")
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I/usr/local/cuda/include",
                        os.path.join(HERE, "arith_host_check.cpp"), "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        assert "failures 0" in r.stdout
