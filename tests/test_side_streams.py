"""Order of a build's launches over its side streams (csrc/cuda/side_streams.cuh),
compiled against a stand-in of the stream calls that tracks which launches a
stream is ordered behind."""
import os
import subprocess

from conftest import ROOT


def test_streams_are_joined_on_every_way_out(tmp_path):
    host = os.path.join(ROOT, "tests", "host")
    exe = str(tmp_path / "side_streams")
    subprocess.run(["g++", "-std=gnu++17", "-O1", "-I" + os.path.join(host, "streams"),
                    "-I" + os.path.join(ROOT, "gtfock_b200", "csrc", "cuda"), os.path.join(host, "side_streams.cpp"),
                    "-o", exe, "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
