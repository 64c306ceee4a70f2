"""Position arithmetic of Distribution layers (csrc/layer_pos.h), compiled for the host: the SNP of every
position a tile reaches, for steps up to 2^31 - 1, and the residue order of the bit rows."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INT_MAX = 2 ** 31 - 1


@pytest.fixture(scope="module")
def pos(tmp_path_factory):
    d = tmp_path_factory.mktemp("pos")
    (d / "pos.cpp").write_text(
        '#include "layer_pos.h"\nextern "C" {\n'
        "int owned(int first, int step, int n, int m) { return fiu::layer_snp(first, fiu::layer_step(step, n), m); }\n"
        "int row(int j, int step, int n) { return fiu::residue_row(j, fiu::layer_step(step, n), n); }\n"
        "int snp(int r, int step, int n) { return fiu::residue_snp(r, fiu::layer_step(step, n), n); }\n"
        "int sample(int step, long long stride) { return fiu::sample_step(step, stride); }\n}\n")
    so = str(d / "pos.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fwrapv", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "fiuncho_gb300", "csrc"), str(d / "pos.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.sample.argtypes = [ctypes.c_int, ctypes.c_longlong]
    return lib


@pytest.mark.parametrize("n", [2, 40, 1150, 2 ** 21 - 1])
@pytest.mark.parametrize("step", [1, 3, 40, 16_900_000, 70_000_000, 2 ** 28, 2 ** 30, INT_MAX])
def test_positions_past_the_last_owned_snp_stay_past_it(pos, n, step):
    for first in {0, 1, n // 2, n - 1}:
        owned = (n - 1 - first) // step + 1
        for m in sorted(set(range(min(owned + 128, 200))) | set(range(max(0, owned - 2), owned + 128))):
            got, want = pos.owned(first, step, n, m), first + step * m
            assert got == want if want < n else got >= n, (first, m, got)


@pytest.mark.parametrize("n", [1, 2, 7, 40, 129])
@pytest.mark.parametrize("step", [1, 2, 3, 7, 39, 40, 41, 129, INT_MAX])
def test_residue_order(pos, n, step):
    order = [j for r in range(min(step, n)) for j in range(r, n, step)]
    assert [pos.snp(r, step, n) for r in range(n)] == order
    assert [pos.row(j, step, n) for j in order] == list(range(n))


@pytest.mark.parametrize("step,stride", [(1, 1), (1, 10 ** 10), (7, 1000), (2 ** 21, 1078), (2 ** 30, 3), (INT_MAX, 2)])
def test_sample_of_prefixes(pos, step, stride):
    got = pos.sample(step, stride)
    assert step <= got <= min(step * stride, INT_MAX) and got % step == 0
    assert step * stride > INT_MAX or got == step * stride
