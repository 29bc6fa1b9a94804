"""The exact evaluation of pooled contenders with few blocks, as on a part of a
GPU: a block then gathers its share in several turns.  Every contender above its
candidate's lower bound is evaluated once, and each candidate keeps the largest
value, the lowest item id on ties."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import build as B  # noqa: E402

pytestmark = pytest.mark.gpu

DRIVER = r"""
#include "fbp_overlap_fast.cuh"
using namespace fbp;
extern "C" int run(int blocks, u32 n, u32 C, u32 K, u32 L, u32 nmax, const float *v, const float *T, u32 *cand, u32 *best_idx,
                   u32 *best_lab, float *best_ll, float *cand_lb, u8 *fallback, u32 *slot, u32 *item, float *hi, u32 *total,
                   u32 cap, u32 *refined, u64 *key) {
    OvArgs A{};
    A.n = n; A.C = C; A.K = K; A.L = L; A.nmax = nmax; A.S = 2 * nmax + 1;
    A.v = v; A.T = T; A.cand = cand; A.best_idx = best_idx; A.best_lab = best_lab; A.best_ll = best_ll;
    A.cand_lb = cand_lb; A.fallback = fallback; A.pool_slot = slot; A.pool_item = item; A.pool_hi = hi;
    A.pool_total = total; A.pool_cap = cap; A.refined = refined; A.best_key = key;
    cudaFuncSetAttribute(k_ov_refine, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ov_refine_smem_bytes());
    k_ov_refine<<<blocks, kRefineThreads, ov_refine_smem_bytes()>>>(A);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("refine")
    src, lib = d / "driver.cu", d / "driver.so"
    src.write_text(DRIVER)
    subprocess.run([B.nvcc_path(), *B.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", B.CSRC, "-I",
                    os.path.join(B.REPO, "include"), "-o", str(lib), str(src)], check=True)
    return ctypes.CDLL(str(lib))


# entries of a block: less than a turn of 256, exactly one, one more, many; the most that share warps
@pytest.mark.parametrize("blocks,m", [(3, 700), (1, 256), (1, 257), (2, 3001), (23, 24576)])
def test_contenders_of_many_turns(driver, blocks, m):
    C, K, L, nmax, n, slots = 2, 3, 17, 9, 900, 40
    S = 2 * nmax + 1
    r = np.random.Generator(np.random.PCG64(m))
    v, T = r.standard_normal((C, n)).astype(np.float32), r.standard_normal((K, C, L)).astype(np.float32)
    cand = r.permutation(slots).astype(np.uint32)
    lab = r.integers(0, K, slots).astype(np.uint32)
    idx = r.integers(2 * L, n - 3 * L, slots).astype(np.uint32)
    ll = r.uniform(-20, 0, slots).astype(np.float32)
    lb = r.uniform(0, 1, slots).astype(np.float32)
    fallback = (r.random(slots) < 0.1).astype(np.uint8)
    slot = r.integers(0, slots, m).astype(np.uint32)
    item = r.integers(0, K * S * S, m).astype(np.uint32)
    hi = r.uniform(0, 2, m).astype(np.float32)
    # values in the reference's order
    w = cand[slot]
    t, a, b = item % K, (item // K) % S, item // (K * S)
    val = np.zeros(m, np.float32)
    for c in range(C):
        ss = np.zeros(m, np.float32)
        for j in range(L):
            jf, js = nmax - a.astype(int) + j, nmax - b.astype(int) + j
            f = np.where((jf >= 0) & (jf < L), T[lab[w], c, np.clip(jf, 0, L - 1)], np.float32(0))
            s = np.where((js >= 0) & (js < L), T[t, c, np.clip(js, 0, L - 1)], np.float32(0))
            x = f + s
            ss = ss + x * x
            val = val + x * v[c, idx[w] + j]
        val = np.where(ss > 0, (val.astype(np.float64) - 0.5 * ss.astype(np.float64)).astype(np.float32), val)
    taken = (fallback[slot] == 0) & ~(hi < lb[slot])
    best = {}
    for e in np.nonzero(taken & (val > ll[w]))[0]:
        g, x = int(slot[e]), (float(val[e]), -int(item[e]))
        best[g] = max(best.get(g, x), x)
    dev = torch.device("cuda", torch.cuda.current_device())
    d = [torch.from_numpy(np.ascontiguousarray(x).view(np.int32) if x.dtype == np.uint32 else x).to(dev)
         for x in (v, T, cand, idx, lab, ll, lb, fallback, slot, item, hi, np.array([m], np.uint32))]
    refined = torch.zeros(1, dtype=torch.int32, device=dev)
    key = torch.zeros(slots, dtype=torch.int64, device=dev)
    p = [ctypes.c_void_p(x.data_ptr()) for x in d]
    assert driver.run(blocks, n, C, K, L, nmax, *p[:12], m, ctypes.c_void_p(refined.data_ptr()),
                      ctypes.c_void_p(key.data_ptr())) == 0
    assert int(refined.item()) == int(taken.sum())
    k = key.cpu().numpy().view(np.uint64)
    for g in range(slots):
        if g not in best:
            assert k[g] == 0
            continue
        u = int(k[g]) >> 32
        bits = u & 0x7fffffff if u & 0x80000000 else ~u & 0xffffffff
        got = (float(np.array([bits], np.uint32).view(np.float32)[0]), -(0xffffffff - (int(k[g]) & 0xffffffff)))
        assert got == best[g], g
