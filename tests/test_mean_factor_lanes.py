"""The mean systems' factorisation kernel under every order of its lanes that the
CUDA execution model allows: the kernel's text, compiled for the host, runs its 32
lanes as coroutines that switch only at the warp-wide operations, in a given order.
A missing barrier between one lane's write and another's read shows as a wrong
factor, or as lanes that wait at different operations.  The reference is the
unblocked band factorisation (DGBTF2) with the reciprocal pivots the kernel keeps;
both sides round every operation in double precision, so the results are equal.
"""
import os
import re
import subprocess

import numpy as np
import pytest

from tests.problems import ROOT

HARNESS = r"""
#include <ucontext.h>
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
using std::max; using std::min; using std::fabs;
#define __global__
#define __launch_bounds__(n)
#define __shared__
struct DevEll {
  int rows, width; const int* cg; const double* val;
  int col(int r, int k) const { return cg[(size_t)k * rows + r]; }
  double v(int r, int k) const { return val[(size_t)k * rows + r]; }
};
struct ZeroSysDev { int T, kl, ku, ldab; DevEll M, L; double* ab; unsigned char* dpiv; };
struct ZeroArgs { int nsys; ZeroSysDev sys[1]; double zsca; int* info; };
struct Index { int x; };
Index threadIdx{0}, blockIdx{0};
double smd[1 << 16];
// ---- lanes: each runs to its next warp-wide operation, in the order given ----
ucontext_t sched, lanes[32];
std::vector<char> stacks[32];
int where[32];   // 0 running, 1 __syncwarp, 2 shuffle, 3 finished
int nshfl[32], cur;
unsigned long long slot[2][32];
void arrive(int kind) {
  const int l = cur;
  where[l] = kind;
  swapcontext(&lanes[l], &sched);
  threadIdx.x = l;
}
void __syncwarp() { arrive(1); }
template <typename T> T __shfl_xor_sync(unsigned, T v, int o) {
  const int l = cur, buf = nshfl[l]++ & 1;
  slot[buf][l] = 0;
  std::memcpy(&slot[buf][l], &v, sizeof v);
  arrive(2);
  T r;
  std::memcpy(&r, &slot[buf][l ^ o], sizeof r);
  return r;
}
@KERNEL@
ZeroArgs g_args; int g_smem;
void lane_main() { k_zero_factor(g_args, g_smem); where[cur] = 3; }
int main(int argc, char** argv) {
  // stdin: T kl ku smem, lane order, rows of M (dense, T x T)
  int T, kl, ku, order[32];
  if (std::scanf("%d %d %d %d", &T, &kl, &ku, &g_smem) != 4) return 2;
  for (int& o : order) if (std::scanf("%d", &o) != 1) return 2;
  std::vector<std::vector<std::pair<int, double>>> rows(T);
  size_t w = 1;
  for (int r = 0; r < T; ++r) {
    for (int c = 0; c < T; ++c) { double v; if (std::scanf("%lf", &v) != 1) return 2; if (v != 0.0) rows[r].push_back({c, v}); }
    w = std::max(w, rows[r].size());
  }
  std::vector<int> cg(w * T, 0); std::vector<double> val(w * T, 0.0);
  for (int r = 0; r < T; ++r) for (size_t k = 0; k < rows[r].size(); ++k) { cg[k * T + r] = rows[r][k].first; val[k * T + r] = rows[r][k].second; }
  const int ldab = 2 * kl + ku + 1;
  std::vector<double> ab((size_t)T * ldab, -7.0); std::vector<unsigned char> piv(T, 99); int info = -1;
  g_args = ZeroArgs{1, {ZeroSysDev{T, kl, ku, ldab, DevEll{T, (int)w, cg.data(), val.data()}, DevEll{T, 0, nullptr, nullptr}, ab.data(), piv.data()}}, 0.0, &info};
  for (int l = 0; l < 32; ++l) {
    stacks[l].resize(1 << 16);
    getcontext(&lanes[l]);
    lanes[l].uc_stack.ss_sp = stacks[l].data(); lanes[l].uc_stack.ss_size = stacks[l].size(); lanes[l].uc_link = &sched;
    makecontext(&lanes[l], lane_main, 0);
  }
  for (bool done = false; !done;) {
    for (int i = 0; i < 32; ++i) { cur = order[i]; threadIdx.x = cur; swapcontext(&sched, &lanes[cur]); }
    for (int l = 1; l < 32; ++l) if (where[l] != where[0]) { std::printf("lanes at different operations\n"); return 1; }
    done = where[0] == 3;
  }
  std::printf("%d\n", info);
  for (int p : piv) std::printf("%d ", p);
  std::printf("\n");
  for (double v : ab) std::printf("%.17g ", v);
  std::printf("\n");
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    with open(os.path.join(ROOT, "coral_b200", "csrc", "kernels.cu")) as f:
        kernel = re.search(r"^__global__ [^\n]*\bk_zero_factor\(.*?^}\n", f.read(), re.S | re.M).group(0)
    d = tmp_path_factory.mktemp("lanes")
    (d / "lanes.cpp").write_text(HARNESS.replace("@KERNEL@", kernel))
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-o", str(d / "lanes"), str(d / "lanes.cpp")], check=True)
    return str(d / "lanes")


def _matrix(T, kl, ku, seed, zero_diagonal):
    rng = np.random.default_rng(seed)
    A = np.zeros((T, T))
    for i in range(T):
        for j in range(max(0, i - kl), min(T, i + ku + 1)):
            A[i, j] = rng.uniform(0.5, 1.5) * rng.choice([-1.0, 1.0])
    if zero_diagonal:
        A[np.arange(0, T - 1, 2), np.arange(0, T - 1, 2)] = 0.0
    return A


def _dgbtf2(A, kl, ku):
    """band storage and pivot offsets of the factorisation, diagonal as reciprocals"""
    T, kv = len(A), kl + ku
    ab, piv, info, ju = np.zeros((T, 2 * kl + ku + 1)), [], 0, 0
    for i in range(T):
        for j in range(T):
            if A[i, j] != 0.0:
                ab[j, kv + i - j] = A[i, j]
    for j in range(T):
        km = min(kl, T - 1 - j)
        jp = int(np.argmax(np.abs(ab[j, kv:kv + km + 1])))
        piv.append(jp)
        if ab[j, kv + jp] == 0.0:
            info = info or j + 1
            continue
        ju = max(ju, min(j + ku + jp, T - 1))
        for c in range(j, ju + 1):
            a, b = kv + j + jp - c, kv + j - c
            ab[c, a], ab[c, b] = ab[c, b], ab[c, a]
        r = 1.0 / ab[j, kv]
        ab[j, kv + 1:kv + km + 1] *= r
        for c in range(j + 1, ju + 1):
            for q in range(1, km + 1):
                ab[c, kv + j + q - c] -= ab[j, kv + q] * ab[c, kv + j - c]
        ab[j, kv] = r
    return info, piv, ab


ORDERS = {"ascending": list(range(32)), "descending": list(range(31, -1, -1)),
          "odd_first": list(range(1, 32, 2)) + list(range(0, 32, 2))}


@pytest.mark.parametrize("order", sorted(ORDERS))
@pytest.mark.parametrize("smem", [0, 1])
@pytest.mark.parametrize("T,kl,ku,kind", [(24, 3, 4, "full"), (24, 3, 4, "zero_diagonal"), (40, 9, 14, "zero_diagonal"),
                                          (5, 3, 4, "zero_diagonal"), (24, 3, 4, "singular")])
def test_lane_orders_agree_with_the_sequential_factorisation(harness, T, kl, ku, kind, smem, order):
    A = _matrix(T, kl, ku, 1, kind != "full")
    if kind == "singular":
        A[:, 0] = 0.0
    words = [T, kl, ku, smem] + ORDERS[order] + ["%.17g" % v for v in A.ravel()]
    r = subprocess.run([harness], input=" ".join(map(str, words)), capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
    info, piv, ab = r.stdout.strip().split("\n")
    ref_info, ref_piv, ref_ab = _dgbtf2(A, kl, ku)
    assert int(info) == ref_info and [int(p) for p in piv.split()] == ref_piv
    assert np.array_equal(np.array(ab.split(), dtype=float), ref_ab.ravel())
