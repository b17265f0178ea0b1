"""The one-block sort of small scenes against the sort over the whole system,
and the rule that chooses between them."""
import itertools
import os
import subprocess

import numpy as np
import pytest

import sph_gb300 as S
from conftest import PKG
from helpers import REF

RULE = r"""
#include <cstdio>
#include "sph_kernels.h"
int main() {
    long long n, k;
    while (scanf("%lld %lld", &n, &k) == 2) printf("%zu %d\n", sph::sort_small_smem(n, k), sph::sort_crowded(n, k));
}
"""
BLOCK = 227 * 1024  # shared memory that a block can have


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    """(shared memory, crowded?) of (particles, keys) pairs."""
    import build

    build.build()
    d = tmp_path_factory.mktemp("rule")
    src, exe = d / "rule.cpp", d / "rule"
    src.write_text(RULE)
    r = subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", f"-I{build.CSRC}", "-I" + os.path.join(PKG, "..", "include"),
                        str(src), os.path.join(build.BUILD, "sph_kernels.cu.o"), "-cudart", "static", "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]

    def ask(sizes):
        out = subprocess.run([str(exe)], input="\n".join(f"{n} {k}" for n, k in sizes), capture_output=True, text=True,
                             check=True).stdout.split()
        return list(zip(map(int, out[::2]), map(int, out[1::2])))

    return ask


def test_rule(rule):
    """At most 4,096 particles and 45,056 keys (key ranges are multiples of 4,096)."""
    sizes = list(itertools.product([1, 4095, 4096, 4097], [4096, 8192, 40960, 45056, 49152, 1 << 20]))
    for (n, k), (smem, _) in zip(sizes, rule(sizes)):
        assert (smem > 0) == (n <= 4096 and k <= 45056), (n, k, smem)
        assert smem == 0 or (4096 + k) * 4 <= smem <= BLOCK - 2048, (n, k, smem)


def test_crowded_cells(rule):
    """More than 16 particles to a key, where a thread has more than two particles."""
    sizes = [(1, 2), (2048, 2), (2049, 2), (2049, 128), (2049, 129), (4096, 255), (4096, 256)]
    assert [c for _, c in rule(sizes)] == [0, 0, 1, 1, 0, 1, 0]


def states(sizes, dims, fill, tile, clump, cell_mult=0.5):
    """Keys, order and state after three steps of scenes with grids of dims
    cells, the second scene stopped after one, beside `fill` other particles."""
    rng = np.random.default_rng(5)
    cell = REF["smoothing_radius"] * 0.5 * (1 + 2.0 ** -12)  # cells of h/2
    half = np.array(dims) * (cell / 2) * 0.9999
    prm = dict(REF, cell_mult=cell_mult, box_half=tuple(half), dt=1e-3)
    out = []
    with S.System(particle_capacity=sum(sizes) + fill, tile=tile) as sysm:
        scenes = []
        for n in sizes:
            sc = sysm.scene(S.default_params(**prm, flags=S.SPH_FLAG_RECORD), capacity=n)
            pos = rng.uniform(-0.95, 0.95, (n, 3)) * half
            pos[: int(n * clump)] = pos[0] + rng.uniform(-1e-3, 1e-3, (int(n * clump), 3))
            sc.set_particles(pos.astype(np.float32), rng.normal(0.0, 0.3, (n, 3)).astype(np.float32))
            scenes.append(sc)
        if fill:
            other = sysm.scene(S.default_params(**dict(REF, box_len=0.4)), capacity=fill)
            other.set_particles(rng.uniform(-0.38, 0.38, (fill, 3)).astype(np.float32))
        for sc in scenes:
            out += [*sc.debug_sort()]
        if len(scenes) > 1:
            scenes[1].set_steps(1)
        sysm.step(3)
        for sc in scenes:
            out += [*sc.get_records(), sc.debug_sort()[1]]
    return out


CASES = [([n], dims) for n in (1, 1025, 4096) for dims in ((2, 3, 4), (35, 33, 39), (44, 32, 32))]  # 45,046 and 45,057 keys
CASES.append(([1, 33, 1000, 4096, 2], (35, 33, 39)))


@pytest.mark.gpu
@pytest.mark.parametrize("clump", [0.0, 0.7])
@pytest.mark.parametrize("tile", [128, 256])
@pytest.mark.parametrize("sizes,dims", CASES)
def test_same_order_and_state(sizes, dims, tile, clump):
    for a, b in zip(states(sizes, dims, 0, tile, clump), states(sizes, dims, 5000, tile, clump)):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2048, 2049, 4096])
@pytest.mark.parametrize("cell_mult", [1.0, 4.0, 8.0])
def test_full_cells(n, cell_mult):
    for a, b in zip(states([n], (16, 16, 16), 0, 256, 0.0, cell_mult), states([n], (16, 16, 16), 5000, 256, 0.0, cell_mult)):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")
