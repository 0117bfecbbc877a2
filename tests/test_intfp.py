"""Binary64 arithmetic on the integer pipe (m2cg_intfp.cuh) and the two forms of
the exact Riemann solver.

CPU: the header compiled for the host, its binary32 hardware estimates replaced
by correctly rounded ones moved by up to their documented error (rcp.approx: 1
ulp; rsqrt.approx: 2^-22.9 relative, two ulps next to 1).  Quotients and roots
must equal the host's IEEE results bit for bit; the reciprocal and the
reciprocal root round a value known to 2^-61 once (at most 0.51 ulp); the
limited slope takes two roundings of a factor in [1, 1.21] and a product (at
most 2 ulp of the exact slope).

GPU: a batch with at most one problem per warp of the launch is solved by the
cooperative solver, a larger one by one thread per problem: the same bits,
stalled solves with the non-adaptive retry included."""
import shutil
import subprocess

import numpy as np
import pytest

from m2c_gb300 import abi, warmstart

import os
HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "m2c_gb300", "csrc",
                      "m2cg_intfp.cuh")

HOST = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
static int pert = 0;
#define M2CG_INT static inline
#define M2CG_INT_SLOW static
namespace m2cg {
static inline uint64_t u64(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
static inline double d64(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
static inline float f32(uint32_t b) { float f; memcpy(&f, &b, 4); return f; }
static inline uint32_t u32(float f) { uint32_t b; memcpy(&b, &f, 4); return b; }
static inline uint32_t if_mulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline uint32_t if_hi(double x) { return (uint32_t)(u64(x) >> 32); }
static inline uint32_t if_lo(double x) { return (uint32_t)u64(x); }
static inline double if_dbl(uint32_t h, uint32_t l) { return d64(((uint64_t)h << 32) | l); }
static inline int if_clz(uint32_t x) { return __builtin_clz(x); }
static inline int clamp1(int p) { return p > 1 ? 1 : p < -1 ? -1 : p; }
static inline uint32_t if_seed_rcp(uint32_t f) { return u32((float)(1.0 / f32(f))) + clamp1(pert); }
static inline uint32_t if_seed_rsqrt(uint32_t f) {
  float y = (float)(1.0 / sqrt((double)f32(f)));
  return u32(y) + (y < 0.9f ? clamp1(pert) : pert);
}
static inline double if_mul(double a, double b) { return a * b; }
static double if_sqrt_slow(double x) { return sqrt(x); }
}
#include "HEADER"
using namespace m2cg;
static uint64_t s = 88172645463325252ull;
static uint64_t nx() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double mk(uint64_t r, int e) { return d64((r & 0x800fffffffffffffull) | ((uint64_t)e << 52)); }
static const uint64_t sig[8] = {0, 1, 2, 0xfffffffffffffull, 0xffffffffffffeull, 0x8000000000000ull, 0x7ffffffffffffull, 0x6a09e667f3bcdull};
static bool same(double a, double b) { return u64(a) == u64(b) || (std::isnan(a) && std::isnan(b)); }
static double ulps(double y, long double ex) { int e; frexp((double)ex, &e); return (double)(fabsl((long double)y - ex) / ldexpl(1.0L, e - 53)); }
int main() {
  long div = 0, root = 0;
  double er = 0, es = 0, ev = 0;
  const double odd[6] = {0.0, -0.0, 4.9e-324, INFINITY, NAN, 1.7e308};
  for (pert = -2; pert <= 2; pert++)
    for (long i = 0; i < 3000000; i++) {
      uint64_t r1 = nx(), r2 = nx(), r3 = nx();
      if (!(r3 & 15)) r1 = (r1 & ~0xfffffffffffffull) | sig[(r3 >> 4) & 7];
      if (!(r3 & 0xf00)) r2 = (r2 & ~0xfffffffffffffull) | sig[(r3 >> 12) & 7];
      double a = mk(r1, 1 + (r3 >> 20) % 2046), b = mk(r2, 1 + (r3 >> 40) % 2046);
      if (i & 1) { a = mk(r1, 1000 + (r3 >> 20) % 46); b = mk(r2, 1000 + (r3 >> 40) % 46); }
      if ((i & 7) == 3) a = b * (double)(1 + (r3 >> 30) % 4096);
      if ((i & 7) == 5) a = b * (1.0 + ((double)(int)((r3 >> 30) & 0xff) - 128) * 0x1p-52);
      if ((i & 1023) == 7) a = odd[r3 % 6];
      if ((i & 1023) == 9) b = odd[r3 % 6];
      div += !same(ddiv(a, b), a / b) + !same(ddiv_lat(a, b), a / b);
      double q, w;
      ddiv2(a, b, b, a, q, w);
      div += !same(q, a / b) + !same(w, b / a);
      double x = fabs(a);
      if ((i & 7) == 5 && b == b) x = b * b;
      root += !same(dsqrt(x), sqrt(x)) + !same(if_sqrt_lat(x), sqrt(x));
      if (if_rcp_range(if_hi(b)) && fabs(b) < 1e300) { double d = ulps(if_rcp_core(if_hi(b), if_lo(b)), 1.0L / b); er = d > er ? d : er; }
      if (if_rsqrt_range(if_hi(x))) { double d = ulps(if_rsqrt_core(if_hi(x), if_lo(x)), 1.0L / sqrtl(x)); es = d > es ? d : es; }
      double p = mk(r1, 960 + (r3 >> 20) % 100), t = mk(r2, 960 + (r3 >> 40) % 100), o;
      if ((i & 63) == 1) t = copysign(1e-16 / fabs(p), p) * (1 + 0x1p-52 * ((int)(r3 >> 56) - 128));
      if (i & 2) t = copysign(p, t) * (1 + 1e-3 * ((r3 >> 50) & 7));
      if (if_van_albada(p, t, o)) {
        const bool zero = p * t <= 0 || fabs(p * t) < 1e-16;
        long double P = p, T = t;
        double d = zero ? (o != 0 ? 1e9 : 0) : ulps(o, (T * P * P + P * T * T) / (P * P + T * T));
        ev = d > ev ? d : ev;
      }
    }
  printf("%ld %ld %.6f %.6f %.6f\n", div, root, er, es, ev);
}
"""


def test_integer_pipe_arithmetic_on_cpu(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "intfp.cpp", tmp_path / "intfp"
    src.write_text(HOST.replace("HEADER", HEADER))
    r = subprocess.run([cc, "-O2", "-std=c++17", "-ffp-contract=off", str(src), "-o", str(exe)], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300).stdout.split()
    assert out[:2] == ["0", "0"]
    er, es, ev = map(float, out[2:])
    # np.longdouble carries 11 bits (x86) or 60 (Arm) beyond binary64's 53
    assert er <= 0.51 and es <= 0.51 and ev <= 2.0


def _problems(n, seed):
    """Interface-like problems of three materials; the last 64 are at equal
    pressures with velocity jumps of 1e-9 m/s, where the secant stalls and the
    non-adaptive retry runs."""
    rng = np.random.default_rng(seed)
    ids = rng.integers(0, 3, (2, n)).astype(np.int32)
    V = np.zeros((2, n, 5))
    V[:, :, 0] = np.choose(ids, [1000.0, 1.2, 1000.0]) * 10.0 ** rng.uniform(-0.15, 0.15, (2, n))
    V[:, :, 1:4] = rng.uniform(-60.0, 60.0, (2, n, 3))
    V[:, :, 4] = np.choose(ids, [1.0e7, 1.0e6, 1.0e7]) * 10.0 ** rng.uniform(-1.0, 1.5, (2, n))
    ids[0, -64:], ids[1, -64:] = 0, 1
    V[0, -64:, 0], V[1, -64:, 0] = 1003.0, 1.2
    V[:, -64:, 4] = 1.0e5
    V[:, -64:, 1:4] = rng.uniform(-1e-9, 1e-9, (2, 64, 3))
    dirs = np.zeros((n, 3))
    dirs[np.arange(n), rng.integers(0, 3, n)] = 1.0
    return V[0], ids[0].copy(), V[1], ids[1].copy(), dirs


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 65, 1216, 1217])
def test_cooperative_solver_equals_one_thread_per_problem(n):
    from m2c_gb300.solver import Solver
    cfg = warmstart.solver_config()
    cfg.n_materials = 3
    abi.set_material(cfg.mat[0], abi.EOS_SG, gamma=6.12, pc=3.43e8)
    abi.set_material(cfg.mat[1], abi.EOS_SG, gamma=1.4, pc=0.0)
    abi.set_material(cfg.mat[2], abi.EOS_NASG, gamma=1.19, pc=6.2e8, b=6.61e-4, q=0.0)
    s = Solver(cfg)
    p = _problems(n, 17)
    few = s.riemann_batch(*p)
    rep = -(-4000 // n)
    many = s.riemann_batch(*[np.concatenate([a] * rep) for a in p])   # more problems than warps
    for k in ("Vs", "id", "Vsm", "Vsp", "iters", "err"):
        np.testing.assert_array_equal(few[k], many[k][:n], err_msg=k)
        np.testing.assert_array_equal(few[k], many[k][-n:], err_msg=k)
    assert few["iters"].max() > 200   # the retry of a stalled solve ran
    s.close()
