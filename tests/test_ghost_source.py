"""The block and cell a copied ghost cell is read at (ghost_copy_src of the stage kernel), on the CPU
against plain division: meshes of so many cells along a direction that a product of a cell index and
a block's width leaves 32 bits."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

import host_math

pytestmark = pytest.mark.skipif(host_math.compiler() is None, reason="no C++ compiler")

# what the function sees of aph_internal.h and aph_amr.cuh
STUBS = r"""
#include "cuda_runtime.h"
constexpr int IV1 = 1, FACE_SAME = 0, FACE_BOUNDARY = 3;
struct AmrFaces { int origin[2], kind[4], nbr[4][4]; };
struct StepBlock { int nx[3], loc[3]; unsigned inv[3][7]; AmrFaces amr; };
struct PackDev { int amr, ng, nb[3], mesh_nx[3], bc[3][2]; };
struct StageArgs { PackDev p; const StepBlock *blocks; };
static long long amr_cell(const StepBlock &, int, int, int, int) { return -1; }
"""

# blocks of a 1D mesh, all of width n; for ghost c of block b: the source block and its cell (first: 0)
BODY = r"""
extern "C" void sources(int nblocks, int n, int lo, int hi, const int *b, const int *c, int count, int *out) {
  StepBlock *blocks = new StepBlock[nblocks]();
  for (int i = 0; i < nblocks; ++i) {
    blocks[i].nx[0] = n, blocks[i].nx[1] = blocks[i].nx[2] = 1, blocks[i].loc[0] = i;
    for (int d = 0; d < 3; ++d)
      for (int k = 0; k < 7; ++k) blocks[i].inv[d][k] = 0xffffffffu / (unsigned)(blocks[i].nx[d] + k) + 1u;
  }
  StageArgs a{};
  a.p.nb[0] = nblocks, a.p.nb[1] = a.p.nb[2] = 1;
  a.p.mesh_nx[0] = nblocks * n;
  a.p.bc[0][0] = lo, a.p.bc[0][1] = hi;
  a.blocks = blocks;
  for (int i = 0; i < count; ++i) {
    const StepBlock *S = nullptr;
    long long sc = -1;
    int flipv = -2;
    ghost_copy_src<1>(a, blocks[b[i]], 0, c[i], 0, 1, S, sc, flipv);
    out[3 * i] = (int)(S - blocks), out[3 * i + 1] = (int)sc, out[3 * i + 2] = flipv;
  }
  delete[] blocks;
}
"""


@pytest.fixture(scope="module")
def sources(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("ghosts"))
    text = ""
    for name in ("aph_window.cuh", "aph_stage.cuh"):
        with open(os.path.join(host_math.CSRC, name)) as f:
            text += f.read()
    parts = [x for p in (
        r"__device__ __forceinline__ int \w+_div\(.*?\n}\n", r"__device__ __forceinline__ int map_index\(.*?\n}\n",
        r"template <int DIR>\n__device__ __forceinline__ bool ghost_copy_src\(.*?\n}\n") for x in re.findall(p, text, re.S)]
    with open(os.path.join(d, "cuda_runtime.h"), "w") as f:
        f.write(host_math.SHIM)
    src, so = os.path.join(d, "g.cpp"), os.path.join(d, "g.so")
    with open(src, "w") as f:
        f.write(STUBS + "".join(parts) + BODY)
    subprocess.check_call([host_math.compiler(), "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-I", d, src, "-o", so])
    return ctypes.CDLL(so).sources


@pytest.mark.parametrize("bc", ["periodic", "outflow", "reflecting"])
@pytest.mark.parametrize("nblocks,n", [(2458, 1324), (6101, 1000), (7627, 800), (40000, 250), (3, 16), (5, 1), (2, 3)])
def test_sources_of_ghost_cells(sources, nblocks, n, bc):
    if bc == "reflecting" and n < 3:
        pytest.skip("three ghost cells do not mirror into fewer")
    b = np.unique(np.concatenate([[0, 1, nblocks // 2, nblocks - 2, nblocks - 1],
                                  np.linspace(0, nblocks - 1, min(nblocks, 500)).astype(int)])).astype(np.int32)
    ghosts = np.array([-3, -2, -1, n, n + 1, n + 2], np.int32)
    bb, cc = np.repeat(b, ghosts.size), np.tile(ghosts, b.size)
    out = np.full((bb.size, 3), -7, np.int32)
    p = ctypes.POINTER(ctypes.c_int)
    code = {"periodic": 0, "outflow": 1, "reflecting": 2}[bc]
    sources(nblocks, n, code, code, bb.ctypes.data_as(p), cc.ctypes.data_as(p), bb.size, out.ctypes.data_as(p))
    g, N = bb.astype(np.int64) * n + cc, nblocks * n
    outside = (g < 0) | (g >= N)
    if bc == "periodic":
        g = g % N
    elif bc == "outflow":
        g = np.clip(g, 0, N - 1)
    else:
        g = np.where(g < 0, -1 - g, np.where(g >= N, 2 * N - 1 - g, g))
    want = np.stack([g // n, g % n, np.where(outside & (bc == "reflecting"), 1, -1)], axis=1)
    assert np.array_equal(out, want), (bb[(out != want).any(axis=1)][:4], out[(out != want).any(axis=1)][:4])


@pytest.mark.gpu
def test_step_of_a_long_mesh():
    """One step of 2,458 blocks of 1,324 cells (3.25e6 in a row) equals the oracle, bit for bit."""
    from apophis_gb300 import problems
    from apophis_gb300.stepper import Stepper
    from oracle import oracle as O
    cfg, cons = problems.sod(nx=2458 * 1324, block_nx=1324, recon="plm", rsolver="hllc", ng=2)
    si = cfg.interior[2]
    cons[:, 0, 0, 0, si] *= 1.0 + 0.25 * np.random.default_rng(8).random(cons[:, 0, 0, 0, si].shape)
    ref = O.Mesh(cfg)
    ref.set_cons(cons)
    ref.run(nsteps=1)
    st = Stepper(cfg, cons, exact=True)
    st.step(1)
    assert np.array_equal(st.state()[:, :, 0, 0, si], ref.get()[:, :, 0, 0, si])
    st.close()
