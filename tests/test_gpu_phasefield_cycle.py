"""The single-block coarse cycle of the Phase-Field solve for 2D levels with even rows (k_mg_vcycle_block_2d) against
the general one (k_mg_vcycle_block): one application to the same right-hand side on the same levels. The two
take the same updates in the same order and differ where the 2D one multiplies by a reciprocal formed once
(h^-2 times the face coefficient, 1/idiag), so they agree to rounding. The kernels have no entry point of their
own; the test compiles the solver's unit with a caller of both."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from compas_b200 import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include "phasefield.cu"
using namespace compas;
extern "C" int cycles(const int* n, const int* per, const double* bx, const double* by, const double* b, const double* x0,
                      int x_zero, double* general, double* rows) {
    compas_b200_parm p;
    compas_b200_geom g;
    memset(&p, 0, sizeof(p));
    memset(&g, 0, sizeof(g));
    p.dim = 2;
    p.physics = COMPAS_B200_FIVEEQS;
    g.n[2] = 1;
    g.ng = 3;
    for (int d = 0; d < 2; ++d) {
        g.n[d] = n[d];
        g.dx[d] = 1.0 / n[0];
        g.lo_bc[d] = g.hi_bc[d] = per[d] ? 0 : 4;
    }
    PfLevel* pf = nullptr;
    std::string err;
    if (pf_create(&p, &g, &pf, &err) != COMPAS_B200_OK) return -1;
    const int nl = (int)pf->mg.size();
    bool ok = pf->mg_block0 == 0 && nl <= kBlk2Levels;
    for (int l = 0; l < nl; ++l) ok = ok && pf->mg[l].rb && pf->mg[l].m.n[0] % 2 == 0;
    const long long nv = pf->mg[0].m.nv;
    if (ok) {
        MgLevel& F = pf->mg[0];
        cudaMemcpy(F.beta[0], bx, sizeof(double) * F.m.nf[0], cudaMemcpyHostToDevice);
        cudaMemcpy(F.beta[1], by, sizeof(double) * F.m.nf[1], cudaMemcpyHostToDevice);
        cudaMemcpy(F.b, b, sizeof(double) * nv, cudaMemcpyHostToDevice);
        for (int l = 1; l < nl; ++l)
            for (int d = 0; d < 2; ++d)
                k_mg_beta<<<blocks_for(pf->mg[l].m.nf[d]), kThreads>>>(pf->mg[l - 1].beta[d], pf->mg[l - 1].m, pf->mg[l].beta[d],
                                                                       pf->mg[l].m, d);
        for (int l = 0; l < nl; ++l) k_mg_idiag<<<blocks_for(pf->mg[l].m.nv), kThreads>>>(pf->mg[l]);
        cudaFuncSetAttribute(k_mg_vcycle_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlockSmemMax);
        cudaFuncSetAttribute(k_mg_vcycle_block_2d, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlockSmemMax);
        for (int k = 0; k < 2; ++k) {
            cudaMemcpy(F.x, x0, sizeof(double) * nv, cudaMemcpyHostToDevice);
            if (k == 0) {
                if (x_zero) cudaMemset(F.x, 0, sizeof(double) * nv);
                k_mg_vcycle_block<<<1, kBlockThreads, pf->mg_block_smem>>>(pf->mg_dev, 0, nl);
            } else {
                k_mg_vcycle_block_2d<<<1, kBlockThreads, pf->mg_block_smem>>>(pf->mg_dev, 0, nl, x_zero);
            }
            cudaMemcpy(k ? rows : general, F.x, sizeof(double) * nv, cudaMemcpyDeviceToHost);
        }
    }
    const cudaError_t e = cudaDeviceSynchronize();
    pf_destroy(pf);
    return !ok ? -2 : e == cudaSuccess ? nl : -3;
}
"""


@pytest.fixture(scope="module")
def cycles(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not found")
    d = tmp_path_factory.mktemp("cycle")
    src, out = os.path.join(d, "cycle.cu"), os.path.join(d, "cycle.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.check_call(["nvcc"] + build.ARCH + build.FLAGS + ["-I" + build.CSRC, "-shared", "-o", out, src])
    return ctypes.CDLL(out).cycles


@pytest.mark.parametrize("x_zero", [1, 0])
@pytest.mark.parametrize("periodic", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("n", [(64, 48), (64, 32), (80, 36), (48, 18), (24, 9), (8, 250), (128, 4), (16, 16), (6, 10), (4, 3)])
def test_the_2d_cycle_is_the_general_cycle(cycles, n, periodic, x_zero):
    sides = [n]
    while all(m % 2 == 0 and m >= 4 for m in sides[-1]) and sides[-1][0] * sides[-1][1] > 16:
        sides.append((sides[-1][0] // 2, sides[-1][1] // 2))
    if any(s[0] % 2 or (periodic[1] and s[1] % 2) for s in sides):
        pytest.skip("odd rows, or a periodic odd side without a two-colour order: the 2D cycle is not taken")
    rng = np.random.default_rng(n[0] + 3 * n[1])
    bx, by = (1e-3 + 10.0 ** rng.uniform(-3, 0, m) for m in ((n[0] + 1) * n[1], n[0] * (n[1] + 1)))
    b, x0 = rng.standard_normal(n[0] * n[1]), rng.standard_normal(n[0] * n[1])
    b -= b.mean()
    out = [np.full(n[0] * n[1], np.nan) for _ in range(2)]
    dp = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    na, pa = np.array(n, dtype=np.int32), np.array(periodic, dtype=np.int32)
    rc = cycles(dp(na), dp(pa), dp(bx), dp(by), dp(b), dp(x0), ctypes.c_int(x_zero), dp(out[0]), dp(out[1]))
    assert rc == len(sides)
    # some 16 sweeps a level, each a few roundings of 2^-53 a cell, amplified at most by the smoother's spectral
    # radius of 1: 1e-12 of the largest value
    diff = np.abs(out[0] - out[1]).max() / np.abs(out[0]).max()
    print(f"{n[0]} x {n[1]}, {rc} levels: {diff:.1e}")
    assert np.isfinite(diff) and diff <= 1e-12
