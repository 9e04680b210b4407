"""Devices that cannot run every thread-block cluster (a partition of a GPU has
fewer SMs together): the library asks how many clusters can be resident and
leaves a cloth whose cluster cannot to another driver.

The library's objects are linked once more with the two runtime calls that know
about clusters replaced by ones that allow eight blocks at most: the occupancy
query answers 0 for a larger cluster, its launch is refused on the host."""
from __future__ import annotations

import shutil
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <cuda_runtime.h>
static int blocks(const cudaLaunchConfig_t *c)
{
    for (unsigned i = 0; i < c->numAttrs; i++)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension)
            return int(c->attrs[i].val.clusterDim.x);
    return 1;
}
extern "C" {
cudaError_t __real_cudaOccupancyMaxActiveClusters(int *, const void *, const cudaLaunchConfig_t *);
cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **);
cudaError_t __wrap_cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c)
{
    *n = 0;
    return blocks(c) > 8 ? cudaSuccess : __real_cudaOccupancyMaxActiveClusters(n, f, c);
}
cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a)
{
    return blocks(c) > 8 ? cudaErrorInvalidClusterSize : __real_cudaLaunchKernelExC(c, f, a);
}
}
"""

CHILD = r"""
import sys
sys.path[:0] = [sys.argv[2], sys.argv[2] + "/tests"]
from pathlib import Path
from acousticsim_gb300 import ClothContext, params
from acousticsim_gb300 import _native as N
N.LIB_PATH = Path(sys.argv[1])
import test_server as T
ctx = ClothContext(0)
p = params(max_iters=5000, rel_tol=T.REL_TOL)
# clusters of 1, 4, 16 (refused) and 16 blocks
work = [(12, 3e2, 3), (40, 1e3, 2), (80, 1e3, 2), (64, 3e2, 2)]
alone = T._twins(ctx, work, p)
served, stats = T._serve(ctx, work, p, budget=4 << 30, max_inflight=0, chunk_iters=8)
T._check_same(served, alone)
# a step of one such cloth, and a set of them
for n in (1, 2):
    cl = [T._cloth(ctx, k, s, 100 + i) for i, (k, s, _) in enumerate(work[2:2 + n], 2)]
    st = ctx.batch_step(cl, 0.0, p)
    assert [s["status"] for s in st] == ["OK"] * n, st
    assert [s["iters"] for s in st] == [alone[2 + i][2][0] for i in range(n)], st
    for c in cl:
        c.close()
ctx.close()
print("served", stats["completed"])
"""


def test_refused_clusters_run_by_other_drivers(built, tmp_path):
    from acousticsim_gb300 import build
    nvcc = build._nvcc()
    objs = sorted(build.BUILD.glob("*.o"))
    assert objs and shutil.which("g++")
    (tmp_path / "shim.cpp").write_text(SHIM)
    inc = Path(nvcc).resolve().parents[1] / "include"
    subprocess.run(["g++", "-O2", "-fPIC", f"-I{inc}", "-c", str(tmp_path / "shim.cpp"), "-o",
                    str(tmp_path / "shim.o")], check=True)
    lib = tmp_path / "libcloth_gb300.so"
    subprocess.run([nvcc, *build.ARCH, "-shared", "-o", str(lib), *map(str, objs),
                    str(tmp_path / "shim.o"), "-lpthread", "-Xlinker",
                    "--wrap=cudaOccupancyMaxActiveClusters,--wrap=cudaLaunchKernelExC"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, str(lib), str(build.ROOT)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "served 9" in r.stdout, r.stdout + r.stderr[-3000:]
