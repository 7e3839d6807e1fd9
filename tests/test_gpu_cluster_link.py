"""The waits of the cluster kernels end, and end the same way for every thread of
a CTA (cluster_link_check.cu, compiled here against the library's header)."""
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("link") / "cluster_link_check"
    nvcc = "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    f"-I{ROOT / 'include'}", f"-I{ROOT / 'tpds22-artifact_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cluster_link_check.cu"), "-o", str(exe)], check=True, capture_output=True)
    return exe


def test_the_check_builds(program):
    assert program.exists()


@pytest.mark.gpu
def test_waits_end_together(ctx, program):
    p = subprocess.run([str(program)], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.startswith("ok"), p.stdout + p.stderr
