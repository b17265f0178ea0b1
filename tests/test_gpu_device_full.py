"""A system whose device memory runs out gives back what it can do without.

The packed records are optional for most variants: they are taken while they
fit.  Calls that a system without them can do must not fail because the system
holds them.  The library's objects are linked once more with a cudaMalloc that
counts bytes and refuses some sizes, or whatever goes above a limit: no device
memory is filled.
"""
import glob
import json
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

FAKE = r"""
#include <cuda_runtime.h>
#include <map>
#include <set>
static std::map<void*, size_t> live;
static std::set<size_t> never;
static size_t total, peak, limit = ~size_t(0);
static int refused;
extern "C" {
cudaError_t __real_cudaMalloc(void**, size_t);
cudaError_t __real_cudaFree(void*);
cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
    if (total + n > limit || never.count(n)) {
        ++refused;
        return cudaErrorMemoryAllocation;
    }
    cudaError_t e = __real_cudaMalloc(p, n);
    if (e == cudaSuccess) {
        live[*p] = n;
        total += n;
        if (total > peak) peak = total;
    }
    return e;
}
cudaError_t __wrap_cudaFree(void* p) {
    auto it = live.find(p);
    if (it != live.end()) {
        total -= it->second;
        live.erase(it);
    }
    return __real_cudaFree(p);
}
void fake_reset(size_t lim) {
    limit = lim;
    never.clear();
    peak = total;
    refused = 0;
}
void fake_never(size_t n) { never.insert(n); }
size_t fake_peak() { return peak; }
int fake_refused() { return refused; }
}
"""

CHILD = r"""
import ctypes as C, hashlib, json, sys
import numpy as np
import sph_gb300 as S
S.LIB_PATH, variant, peak_at = sys.argv[1], int(sys.argv[2]), sys.argv[3]
L = S.lib()
L.fake_reset.argtypes = L.fake_never.argtypes = [C.c_size_t]
L.fake_peak.restype = C.c_size_t
from helpers import REF
CAPS = (24576, 40960)  # the arena has 24,576 entries, then 65,536
RECORDS = [32 * CAPS[0], 32 * sum(CAPS)]
rng = np.random.default_rng(2)
# fewer particles than capacity: no other buffer has the records' size
pos = [rng.uniform(-0.35, 0.35, (n - 100, 3)).astype(np.float32) for n in CAPS]
prm = S.default_params(**dict(REF, box_len=0.4))

def mesh(sysm, sc):
    verts = np.zeros((1500 * 1500, 6), np.float32)
    fn = L.sph_scene_terrain_mesh
    fn.restype, fn.argtypes = C.c_int, [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    assert fn(sysm.h, sc.id, C.c_void_p(verts.ctypes.data), None) == 0, L.sph_last_error()
    return verts.tobytes()

def sequence(limit=2 ** 62, never=()):
    L.fake_reset(limit)
    for n in never:
        L.fake_never(n)
    h = hashlib.sha256()
    with S.System(particle_capacity=CAPS[0], variant=variant) as sysm:
        scenes = []
        for k in range(2):
            scenes.append(sysm.scene(prm, capacity=CAPS[k], terrain=(64, 64)))
            scenes[k].set_particles(pos[k])
            sysm.step(2)
        if peak_at != "lists":
            scenes[1].set_terrain(np.zeros((1500, 1500), np.float32))
            sysm.step(2)
        if peak_at == "mesh":
            h.update(mesh(sysm, scenes[1]))
            sysm.step(2)
        mem = sysm.memory()
        for sc in scenes:
            st = sc.get_particles()
            h.update(st["pos"].tobytes() + st["vel"].tobytes() + st["density"].tobytes())
    return dict(hash=h.hexdigest(), memory=mem, peak=L.fake_peak(), refused=L.fake_refused())

free = sequence()
lean = sequence(never=RECORDS)
tight = sequence(limit=lean["peak"])
json.dump(dict(free=free, lean=lean, tight=tight, records=RECORDS), sys.stdout)
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    import build

    build.build()
    d = tmp_path_factory.mktemp("fake")
    src, lib = str(d / "fake.cpp"), str(d / "libsph_fake.so")
    with open(src, "w") as f:
        f.write(FAKE)
    r = subprocess.run([build.nvcc(), *build.ARCH, "-shared", "-Xcompiler", "-fPIC", "-cudart", "static", "-Xlinker",
                        "--wrap=cudaMalloc,--wrap=cudaFree", "-o", lib, src,
                        *sorted(glob.glob(os.path.join(build.BUILD, "*.o"))), "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return lib


@pytest.mark.parametrize("peak_at", ["lists", "terrain", "mesh"])
@pytest.mark.parametrize("variant", [88, 163960])
def test_optional_records_make_way(library, variant, peak_at):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([PKG, os.path.join(ROOT, "tests")]))
    r = subprocess.run([sys.executable, "-c", CHILD, library, str(variant), peak_at], env=env, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    got = json.loads(r.stdout)
    free, lean, tight = got["free"], got["lean"], got["tight"]
    # with room the records are held, refused they are not, the bits the same
    assert free["refused"] == 0 and lean["refused"] >= 2
    assert free["memory"] - lean["memory"] == got["records"][1]
    assert free["hash"] == lean["hash"]
    # and no more memory than without them suffices
    assert tight["peak"] <= lean["peak"] and tight["hash"] == lean["hash"]
    assert tight["refused"] > 0 or peak_at == "lists"  # the lists' growth releases the records beforehand
