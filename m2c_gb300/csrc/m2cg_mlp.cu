// Learned warm start for the exact two-material Riemann solve: a
// 16 -> 64 -> 64 -> 64 -> 1 SiLU MLP that predicts the star pressure from the
// two states and their EOS parameters.  The exact solver starts from a pair
// bracketing the prediction (in place of the acoustic pair,
// ExactRiemannSolverBase.cpp:1107-1158) and still converges to the same
// tolerance, so its answer, not the prediction, is the result.
//
// The three 64-wide layers run on the tensor cores: tcgen05.mma with BF16
// operands staged in shared memory and FP32 accumulators in tensor memory, one
// 128-row tile per CTA pass.  The scalar head (64 -> 1), biases, SiLU, the
// loss and Adam run on the CUDA cores in FP32.  Training runs forward and
// backward for a tile in one kernel and accumulates the weight gradients with
// FP32 atomics; Adam then updates the FP32 master weights and the BF16 copies
// the GEMMs read.
//
// A tile is a short serial chain (three GEMMs of 2 x 128 x 64 x 64 operations
// and their epilogues, eight in training), so the time is latency: of the
// shared-memory traffic around the GEMMs, the activations and the barriers.
// 16 warps share a tile, each thread holding one row's 16 columns: one 64-byte
// TMEM load per layer, two 16-byte stores into the operand tile, which the
// next GEMM reads K-major and the weight-gradient GEMM, transposed by its
// descriptor, M-major from the same bytes.  SiLU' is kept in registers from
// the forward pass, column sums are taken while the GEMMs run.  A training batch
// of 16,384 rows takes 14 us, a forward pass over 262,144 rows 61 us (94 and
// 216 us with one row per thread, element-wise stores, transposed copies and 320
// shuffles a row for the column sums).
//
// Inputs are dimensionless groups of the two states relative to the
// impedance-weighted pressure p_ref = (C_r p_l + C_l p_r) / (C_l + C_r), with
// c^2 = gamma (p + pc) / (rho (1 - b rho)) and C = rho c (12 used, padded to 16):
//   asinh(a) / 4 with a = (u_l - u_r) C_l C_r / ((C_l + C_r) p_ref), the
//     acoustic pressure jump;
//   ln(p_l / p_ref) / 4, ln(p_r / p_ref) / 4, ln(C_l / C_r) / 4;
//   (gamma_s - 4) / 1.7, asinh(pc_s / p_ref) / 8, 2 b_s rho_s - 1,
//     ln(rho_s c_s^2 / p_ref) / 4 for each side s.
// Target: t = ln(p* / p_ref) / 4, i.e. p* = p_ref exp(4 t).  (Pressures below
// 1 Pa enter the inputs as 1 Pa.)
#include <cstdio>
#include <cstring>
#include <cmath>
#include <vector>
#include <random>
#include <algorithm>
#include <mutex>
#include "m2cg_internal.h"
#include "m2cg_umma.cuh"

void m2cg_set_error(const char* fmt, ...);

#define MCK(call)                                                                                  \
  do {                                                                                             \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess) {                                                                       \
      m2cg_set_error("%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
      return M2CG_ERR_CUDA;                                                                        \
    }                                                                                              \
  } while (0)

namespace m2cg {
namespace mlp {

constexpr int NF = M2CG_MLP_FEATURES;  // 16
constexpr int NH = 64;
constexpr int TILE = 128;
// flat FP32 parameter vector: W1 [64][16], b1, W2 [64][64], b2, W3 [64][64], b3, w4 [64], b4
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NH * NF, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH,
              OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NH * NH, OFF_W4 = OFF_B3 + NH, OFF_B4 = OFF_W4 + NH,
              NPARAM = OFF_B4 + 1;
static_assert(NPARAM == M2CG_MLP_PARAMS, "parameter count");
// BF16 GEMM operands: W1f [64][16], W2f, W3f [64][64] (out x in, the forward
// B operands) and W2b, W3b [64][64] (in x out, the backward B operands), each
// in the operand layout of shared memory, so that a CTA's copy is one run of
// 16-byte words
constexpr int BF_W1F = 0, BF_W2F = BF_W1F + NH * NF, BF_W3F = BF_W2F + NH * NH, BF_W2B = BF_W3F + NH * NH,
              BF_W3B = BF_W2B + NH * NH, NBF = BF_W3B + NH * NH;

constexpr long long MAX_POLLS = 1ll << 26;  // mbarrier wait limit (the MMAs take microseconds)

// Threads of a tile: row r = thread % 128 (the TMEM lane its warp can reach),
// columns 16 (thread / 128) .. + 15.
constexpr int NTHR = 512;
constexpr int CG = 16;         // columns per thread
constexpr int NGRP = NH / CG;  // column groups
static_assert(NTHR == TILE * NGRP, "one thread per row and column group");

// shared-memory layout of the tile kernels (byte offsets, 1024-aligned): the
// weights as in global memory, the operand tiles, then floats.  As the M-major
// operand of a weight-gradient GEMM a tile is read as 128 features, of which
// it has 64 (or 16): the rest, up to 1,792 bytes behind its end, only reach
// accumulator rows that nobody reads.
constexpr int S_W = 0, S_XA = S_W + 2 * NBF, S_H1A = S_XA + 4096, S_H2A = S_H1A + 16384,
              S_FWD_END = S_H2A + 16384, S_DZ3 = S_FWD_END, S_DZ2 = S_DZ3 + 16384, S_DZ1 = S_DZ2 + 16384,
              S_TRAIN_END = S_DZ1 + 16384;
static_assert(S_XA % 1024 == 0, "tile alignment");
// the last hidden layer's activations [64][128] in FP32 for the head: where the
// operand tiles are free at that time
constexpr int S_H3_FWD = S_H1A, S_H3_TRAIN = S_DZ2;
// floats behind them: b1 b2 b3 w4 (4 x 64), b4, padding; in training the rows'
// outputs, the column sums of the four warps of each column: db1 db2 db3 dw4,
// then loss and db4 of the warps of group 0
constexpr int F_B4 = 256, F_OUT = 260, F_SUM = F_OUT + TILE, F_LOSS = F_SUM + 4 * 4 * NH, F_END = F_LOSS + 8;
constexpr int SMEM_FWD = S_FWD_END + F_OUT * 4;
constexpr int SMEM_TRAIN = S_TRAIN_END + F_END * 4;

// s = 1 / (1 + exp(-z)) and z / (1 + exp(-z)), the latter from z s by two exact
// residuals (the first makes it faithful, the second correctly rounded:
// Markstein, IBM J. Res. Dev. 34, 1990); where the residual is no number (an
// infinity) z s is the quotient.
__device__ __forceinline__ float silu(float z, float& s) {
  const float d = 1.0f + expf(-z);
  s = __frcp_rn(d);
  float q = z * s, r = fmaf(-q, d, z);
  if (r == r) {
    q = fmaf(r, s, q);
    q = fmaf(fmaf(-q, d, z), s, q);
  }
  return q;
}
__device__ __forceinline__ float dsilu(float z, float s) { return s * (1.0f + z * (1.0f - s)); }

// ---- features ---------------------------------------------------------------
// f[0..15] and p_ref of one problem: states (rho, u, p) per side, EOS rows
// {type, gamma, pc, b, q}.  Bound by the binary64 pipe (64 cycles per warp
// instruction and sub-partition; five logarithms, three asinh): the ten
// quotients and two roots run on the integer pipe instead, rounded alike, and a
// row leaves in two 16-byte stores (262,144 problems 258 -> 199 us).
__device__ double problem_features(double rl, double ul, double pl, const double* el, double rr, double ur,
                                   double pr, const double* er, float* f) {
  pl = fmax(pl, 1.0);
  pr = fmax(pr, 1.0);
  double c2l = ddiv(el[1] * (pl + el[2]), rl * (1.0 - el[3] * rl));
  double c2r = ddiv(er[1] * (pr + er[2]), rr * (1.0 - er[3] * rr));
  c2l = c2l > 0.0 ? c2l : 1.0;
  c2r = c2r > 0.0 ? c2r : 1.0;
  double Cl = rl * dsqrt(c2l), Cr = rr * dsqrt(c2r);
  double pref = ddiv(Cr * pl + Cl * pr, Cl + Cr);
  double a = ddiv((ul - ur) * Cl * Cr, (Cl + Cr) * pref);
  f[0] = (float)(asinh(a) * 0.25);
  f[1] = (float)(log(ddiv(pl, pref)) * 0.25);
  f[2] = (float)(log(ddiv(pr, pref)) * 0.25);
  f[3] = (float)(log(ddiv(Cl, Cr)) * 0.25);
  f[4] = (float)ddiv(el[1] - 4.0, 1.7);
  f[5] = (float)ddiv(er[1] - 4.0, 1.7);
  f[6] = (float)(asinh(ddiv(el[2], pref)) * 0.125);
  f[7] = (float)(asinh(ddiv(er[2], pref)) * 0.125);
  f[8] = (float)(2.0 * el[3] * rl - 1.0);
  f[9] = (float)(2.0 * er[3] * rr - 1.0);
  f[10] = (float)(log(ddiv(rl * c2l, pref)) * 0.25);
  f[11] = (float)(log(ddiv(rr * c2r, pref)) * 0.25);
  for (int i = 12; i < NF; i++) f[i] = 0.f;
  return pref;
}

// A row of 16 features -> bf16, two 16-byte stores.
__device__ __forceinline__ void put_row(__nv_bfloat16* X, int64_t row, const float* f) {
  uint4 w[2];
  uint32_t* u = reinterpret_cast<uint32_t*>(w);
#pragma unroll
  for (int i = 0; i < NF / 2; i++) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    u[i] = *reinterpret_cast<const uint32_t*>(&b);
  }
  uint4* x = reinterpret_cast<uint4*>(X) + row * 2;
  x[0] = w[0];
  x[1] = w[1];
}

// 1D problems: W rows {rho_l, u_l, p_l, rho_r, u_r, p_r}, E rows {type, gamma,
// pc, b, q} x 2.  X: n x 16 bf16; pref: n; t (optional): targets from pstar.
__global__ void k_features(int64_t n, const double* __restrict__ W, const double* __restrict__ E,
                           const double* __restrict__ pstar, __nv_bfloat16* X, float* pref, float* t) {
  int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const double* w = &W[q * 6];
  float f[NF];
  double pr = problem_features(w[0], w[1], w[2], &E[q * 10], w[3], w[4], w[5], &E[q * 10 + 5], f);
  put_row(X, q, f);
  if (pref) pref[q] = (float)pr;
  if (t && pstar) t[q] = (float)(log(fmax(pstar[q], 1e-300) / pr) * 0.25);
}

// Interface faces of the finite-volume step: inputs as the interface solve
// reads them (cell-centre states, Constant reconstruction at the interface),
// normal velocity along the face's axis.
__global__ void k_features_faces(Params P, StateSet S, const int32_t* __restrict__ id, const IfaceList L,
                                 __nv_bfloat16* X, float* pref, const DevScalars* sc) {
  if (sc && !sc->active) return;
  int64_t n = (int64_t)min((unsigned long long)L.cap, *L.count);
  const int64_t st[3] = {1, P.g.sy, P.g.sz};
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
    int64_t fc = L.face[s];
    int d = (int)(fc & 3);
    int64_t c = fc >> 2, m = c - st[d];
    const DevMat& ML = P.mats.m[id[m]];
    const DevMat& MR = P.mats.m[id[c]];
    double el[5] = {(double)ML.type, ML.gam, ML.Pstiff, ML.type == M2CG_EOS_NASG ? ML.b : 0.0, 0.0};
    double er[5] = {(double)MR.type, MR.gam, MR.Pstiff, MR.type == M2CG_EOS_NASG ? MR.b : 0.0, 0.0};
    float f[NF];
    double pr = problem_features(S.q[0][m], S.q[1 + d][m], S.q[4][m], el, S.q[0][c], S.q[1 + d][c], S.q[4][c], er, f);
    put_row(X, s, f);
    pref[s] = (float)pr;
  }
}

// Network output -> starting pressure p_ref exp(4 t) (0 = no warm start).
__global__ void k_to_pressure(int64_t n, const float* __restrict__ t, const float* __restrict__ pref, double* pd,
                              float* pf, const DevScalars* sc, const unsigned long long* count) {
  if (sc && !sc->active) return;
  if (count) n = min((unsigned long long)n, *count);
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    double p = (double)pref[q] * exp(4.0 * (double)t[q]);
    if (!(p > 0.0) || !(p < 1e300)) p = 0.0;
    if (pd) pd[q] = p;
    if (pf) pf[q] = (float)p;
  }
}

// ---- tile machinery -----------------------------------------------------------
struct TileCtx {
  unsigned char* sm;
  float* f32;
  uint64_t* bar;
  uint32_t tm;
  uint32_t phase;
  bool ok;
  int r, g, j0;   // this thread's row, column group and first column
};

__device__ __forceinline__ void load_weights(TileCtx& c, const __nv_bfloat16* __restrict__ wbf,
                                             const float* __restrict__ prm, bool backward) {
  const int t = threadIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(wbf);
  uint4* dst = reinterpret_cast<uint4*>(c.sm + S_W);
  const int n = (backward ? NBF : BF_W2B) / 8;
  for (int i = t; i < n; i += NTHR) dst[i] = src[i];
  if (t < 256) {
    const int off[4] = {OFF_B1, OFF_B2, OFF_B3, OFF_W4};
    c.f32[t] = prm[off[t >> 6] + (t & 63)];
  }
  if (t == 0) c.f32[F_B4] = prm[OFF_B4];
}

// Orders generic shared-memory writes before MMAs issued after the barrier,
// and TMEM reads before MMAs that overwrite the same columns.
__device__ __forceinline__ void sync_for_mma() {
  umma::fence_async_smem();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
}

// Waits for the MMAs up to the last commit.
__device__ __forceinline__ void wait_mma(TileCtx& c) {
  c.ok = umma::mbar_wait(c.bar, c.phase, MAX_POLLS) && c.ok;
  c.phase ^= 1u;
  umma::fence_after_sync();
}

// TMEM address of this thread's row (lane) at column col + j0.
__device__ __forceinline__ uint32_t trow(const TileCtx& c, int col) {
  return c.tm + ((uint32_t)(c.r & ~31) << 16) + (uint32_t)(col + c.j0);
}

// 16 values of this thread's row and columns -> bf16 in a [128][64] operand tile.
__device__ __forceinline__ void store16(const TileCtx& c, unsigned char* tile, const float (&h)[CG]) {
#pragma unroll
  for (int q = 0; q < 2; q++) {
    uint4 w;
    uint32_t* u = reinterpret_cast<uint32_t*>(&w);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(h[8 * q + 2 * i], h[8 * q + 2 * i + 1]);
      u[i] = *reinterpret_cast<const uint32_t*>(&b);
    }
    *reinterpret_cast<uint4*>(tile + umma::kmajor_offset(c.r, c.j0 + 8 * q, NH)) = w;
  }
}

// Half a network input row (8 features, 16 bytes) per thread of the first 256.
__device__ __forceinline__ uint4 read_x(const __nv_bfloat16* __restrict__ X, int64_t row, bool valid) {
  return valid ? reinterpret_cast<const uint4*>(X)[row * 2 + (threadIdx.x & 1)] : make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void store_x(const TileCtx& c, uint4 x) {
  *reinterpret_cast<uint4*>(c.sm + S_XA + umma::kmajor_offset(threadIdx.x >> 1, (threadIdx.x & 1) * 8, NF)) = x;
}

// Hidden layer l (0, 1): its GEMM, then H = bf16(SiLU(Z + b)) into the operand
// tile dst; ds: SiLU'(Z + b) of this thread's row and columns (training).
template <bool Train>
__device__ __forceinline__ void hidden_layer(TileCtx& c, int l, const unsigned char* in, const unsigned char* w, int K,
                                             unsigned char* dst, float (&ds)[CG]) {
  sync_for_mma();
  if (threadIdx.x == 0) {
    umma::gemm_128xN(c.tm + 64 * l, in, w, NH, K, false);
    umma::mma_commit(c.bar);
  }
  wait_mma(c);
  float v[CG];
  umma::tmem_ld16(trow(c, 64 * l), v);
  const float* b = c.f32 + 64 * l + c.j0;
#pragma unroll
  for (int i = 0; i < CG; i++) {
    const float z = v[i] + b[i];
    float s;
    v[i] = silu(z, s);
    if (Train) ds[i] = dsilu(z, s);
  }
  store16(c, dst, v);
}

// The network for the tile in S_XA: returns, in the threads of group 0, the
// output of the row (the scalar head out = b4 + sum_j SiLU(z3_j + b3_j) w4_j,
// summed in this order by one thread); in training h3, ds1..ds3 of the row's 16
// columns as well.
template <bool Train>
__device__ __forceinline__ float forward_tile(TileCtx& c, float (&h3)[CG], float (&ds1)[CG], float (&ds2)[CG],
                                              float (&ds3)[CG]) {
  const unsigned char* w = c.sm + S_W;
  hidden_layer<Train>(c, 0, c.sm + S_XA, w + 2 * BF_W1F, NF, c.sm + S_H1A, ds1);
  hidden_layer<Train>(c, 1, c.sm + S_H1A, w + 2 * BF_W2F, NH, c.sm + S_H2A, ds2);
  sync_for_mma();
  if (threadIdx.x == 0) {
    umma::gemm_128xN(c.tm + 128, c.sm + S_H2A, w + 2 * BF_W3F, NH, NH, false);
    umma::mma_commit(c.bar);
  }
  wait_mma(c);
  umma::tmem_ld16(trow(c, 128), h3);
  float* hb = reinterpret_cast<float*>(c.sm + (Train ? S_H3_TRAIN : S_H3_FWD)) + c.r;
#pragma unroll
  for (int i = 0; i < CG; i++) {
    const float z = h3[i] + c.f32[128 + c.j0 + i];
    float s;
    h3[i] = silu(z, s);
    if (Train) ds3[i] = dsilu(z, s);
    hb[(c.j0 + i) * TILE] = h3[i];
  }
  __syncthreads();
  float out = c.f32[F_B4];
  if (c.g == 0) {
#pragma unroll 16
    for (int j = 0; j < NH; j++) out = fmaf(hb[j * TILE], c.f32[192 + j], out);
  }
  return out;
}

__device__ __forceinline__ void tile_setup(TileCtx& c, unsigned char* sm, float* f32, uint64_t* bar, uint32_t* tslot) {
  c.sm = sm;
  c.f32 = f32;
  c.bar = bar;
  c.phase = 0;
  c.ok = true;
  c.r = threadIdx.x & (TILE - 1);
  c.g = threadIdx.x / TILE;
  c.j0 = CG * c.g;
  if (threadIdx.x == 0) umma::mbar_init(bar, 1);
  if (threadIdx.x < 32) umma::tmem_alloc(tslot, 256);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  c.tm = *tslot;
}

__device__ __forceinline__ void tile_teardown(TileCtx& c) {
  umma::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) umma::tmem_dealloc(c.tm, 256);
}

// ---- inference ----------------------------------------------------------------
// Persistent: CTA b handles tiles b, b + grid, ...  out[row] = network output.
// rows = min(n, *count) when count is given (the device-side interface count).
// Two CTAs per SM (256 TMEM columns each), one working while the other waits;
// the next tile's inputs are fetched during the current one.
__global__ void __launch_bounds__(NTHR, 2) k_forward(int64_t n, const unsigned long long* count,
                                                      const __nv_bfloat16* __restrict__ X,
                                                      const __nv_bfloat16* __restrict__ wbf,
                                                      const float* __restrict__ prm, float* out, int* err,
                                                      const DevScalars* sc) {
  if (sc && !sc->active) return;
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tslot;
  if (count) n = (int64_t)min((unsigned long long)n, *count);
  int64_t ntiles = (n + TILE - 1) / TILE;
  if ((int64_t)blockIdx.x >= ntiles) return;
  TileCtx c;
  tile_setup(c, sm, reinterpret_cast<float*>(sm + S_FWD_END), &bar, &tslot);
  const bool loads = threadIdx.x < 2 * TILE;
  int64_t xrow = (int64_t)blockIdx.x * TILE + (threadIdx.x >> 1);
  uint4 x = read_x(X, xrow, loads && xrow < n);
  load_weights(c, wbf, prm, false);
  for (int64_t tile = blockIdx.x; tile < ntiles && c.ok; tile += gridDim.x) {
    if (loads) store_x(c, x);
    xrow += (int64_t)gridDim.x * TILE;
    x = read_x(X, xrow, loads && xrow < n);
    float h3[CG], none[CG];
    const float o = forward_tile<false>(c, h3, none, none, none);
    const int64_t row = tile * TILE + c.r;
    if (c.g == 0 && row < n) out[row] = o;
    c.ok = __syncthreads_and(c.ok);   // (also: the head's activations are read)
  }
  if (!c.ok && threadIdx.x == 0) atomicExch(err, 1);
  tile_teardown(c);
}

// ---- training -------------------------------------------------------------------
// Sums of v[0..15] over the 32 rows of the warp into s[0..15]: each step of
// the butterfly also halves the columns a lane keeps, 16 shuffles in all.
__device__ __forceinline__ void col_sums(float* s, const float (&v)[CG]) {
  const int lane = threadIdx.x & 31;
  float a[CG];
#pragma unroll
  for (int i = 0; i < CG; i++) a[i] = v[i];
#pragma unroll
  for (int n = CG / 2, o = 16; n > 0; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; i++) {
      const float give = up ? a[i] : a[i + n], keep = up ? a[i + n] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
  if ((lane & 1) == 0) s[lane >> 1] = a[0];
}

// Weight-gradient readout: 64 TMEM columns from col on hold D[i][j] for input
// feature i = row (< n_in); grad[off + j * n_in + i] += D[i][j].
__device__ __forceinline__ void dw_readout(const TileCtx& c, int col, float* grad, int off, int n_in) {
  if ((c.r & ~31) >= n_in) return;  // warp-uniform: no rows of interest in this warp
  float v[CG];
  umma::tmem_ld16(trow(c, col), v);
  if (c.r < n_in) {
#pragma unroll
    for (int q = 0; q < CG; q++) atomicAdd(&grad[off + (c.j0 + q) * n_in + c.r], v[q]);
  }
}

// One 128-row tile of the batch: forward, squared-error loss on the target,
// backward; gradients (of the mean loss over the batch) and the loss sum are
// accumulated into grad[] and loss[0].  TMEM columns: Z1 0, Z2 64, Z3 128; then
// dW3 192, dH2 128, dW2 0, dH1 64, dW1 128.  Each layer's input gradient is
// issued and committed before its weight gradient, which runs on while the next
// layer's dZ is computed (its own operand tile) and is read after the next wait.
__global__ void __launch_bounds__(NTHR, 1) k_train(int64_t batch, const int32_t* __restrict__ idx,
                                                    const __nv_bfloat16* __restrict__ X, const float* __restrict__ y,
                                                    const __nv_bfloat16* __restrict__ wbf,
                                                    const float* __restrict__ prm, float* grad, float* loss,
                                                    int* err) {
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tslot;
  TileCtx c;
  tile_setup(c, sm, reinterpret_cast<float*>(sm + S_TRAIN_END), &bar, &tslot);
  const int64_t b0 = (int64_t)blockIdx.x * TILE;
  uint4 x = make_uint4(0, 0, 0, 0);
  if (threadIdx.x < 2 * TILE) {
    const int64_t xb = b0 + (threadIdx.x >> 1);
    x = read_x(X, xb < batch ? (idx ? (int64_t)idx[xb] : xb) : 0, xb < batch);
  }
  const bool valid = b0 + c.r < batch;
  const float target = valid ? y[idx ? (int64_t)idx[b0 + c.r] : b0 + c.r] : 0.f;
  load_weights(c, wbf, prm, true);
  if (threadIdx.x < 2 * TILE) store_x(c, x);
  float h3[CG], ds1[CG], ds2[CG], ds3[CG];
  const float o = forward_tile<true>(c, h3, ds1, ds2, ds3);
  if (c.g == 0) c.f32[F_OUT + c.r] = o;
  __syncthreads();
  const float e = valid ? c.f32[F_OUT + c.r] - target : 0.f;
  const float d = 2.f * e / (float)batch;
  const int lane = threadIdx.x & 31, wr = c.r >> 5;
  float* sums = c.f32 + F_SUM + wr * NH + c.j0;   // + 4 NH per quantity
  // layer 3: dZ3 = d w4 SiLU'(z3); dw4 = sum d h3
  float dz[CG];
#pragma unroll
  for (int q = 0; q < CG; q++) {
    dz[q] = d * c.f32[192 + c.j0 + q] * ds3[q];
    h3[q] *= d;
  }
  store16(c, sm + S_DZ3, dz);
  sync_for_mma();
  if (threadIdx.x == 0) {
    umma::gemm_128xN(c.tm + 128, sm + S_DZ3, sm + S_W + 2 * BF_W3B, NH, NH, false);   // dH2[r][i]
    umma::mma_commit(c.bar);
    umma::gemm_tn_128xN(c.tm + 192, sm + S_H2A, NH, sm + S_DZ3, NH, TILE);            // dW3[i][j]
  }
  col_sums(sums + 2 * 4 * NH, dz);
  col_sums(sums + 3 * 4 * NH, h3);
  if (c.g == 0) {
    float l = e * e, db = d;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      l += __shfl_xor_sync(0xffffffffu, l, o);
      db += __shfl_xor_sync(0xffffffffu, db, o);
    }
    if (lane == 0) { c.f32[F_LOSS + wr] = l; c.f32[F_LOSS + 4 + wr] = db; }
  }
  wait_mma(c);
  // layer 2: dZ2 = dH2 SiLU'(z2)
  umma::tmem_ld16(trow(c, 128), dz);
#pragma unroll
  for (int q = 0; q < CG; q++) dz[q] *= ds2[q];
  store16(c, sm + S_DZ2, dz);
  sync_for_mma();
  if (threadIdx.x == 0) {
    umma::gemm_128xN(c.tm + 64, sm + S_DZ2, sm + S_W + 2 * BF_W2B, NH, NH, false);    // dH1
    umma::mma_commit(c.bar);
    umma::gemm_tn_128xN(c.tm + 0, sm + S_H1A, NH, sm + S_DZ2, NH, TILE);              // dW2
  }
  col_sums(sums + 1 * 4 * NH, dz);
  wait_mma(c);
  // layer 1: dZ1 = dH1 SiLU'(z1)
  umma::tmem_ld16(trow(c, 64), dz);
#pragma unroll
  for (int q = 0; q < CG; q++) dz[q] *= ds1[q];
  store16(c, sm + S_DZ1, dz);
  sync_for_mma();
  if (threadIdx.x == 0) {
    umma::gemm_tn_128xN(c.tm + 128, sm + S_XA, NF, sm + S_DZ1, NH, TILE);             // dW1
    umma::mma_commit(c.bar);
  }
  col_sums(sums, dz);
  dw_readout(c, 192, grad, OFF_W3, NH);   // complete: committed with dH1
  wait_mma(c);
  dw_readout(c, 0, grad, OFF_W2, NH);
  dw_readout(c, 128, grad, OFF_W1, NF);
  __syncthreads();
  if (threadIdx.x < 256) {
    const int k = threadIdx.x >> 6, j = threadIdx.x & 63;
    const int off[4] = {OFF_B1, OFF_B2, OFF_B3, OFF_W4};
    const float* s = c.f32 + F_SUM + k * 4 * NH + j;
    atomicAdd(&grad[off[k] + j], (s[0] + s[NH]) + (s[2 * NH] + s[3 * NH]));
  } else if (threadIdx.x < 258) {
    const float* s = c.f32 + F_LOSS + 4 * (threadIdx.x - 256);
    atomicAdd(threadIdx.x == 256 ? loss : &grad[OFF_B4], (s[0] + s[1]) + (s[2] + s[3]));
  }
  if (!c.ok) atomicExch(err, 1);
  tile_teardown(c);
}

// Where parameter i is a GEMM weight: its BF16 copies (forward and transposed).
__device__ __forceinline__ void pack_param(int i, float v, __nv_bfloat16* wbf) {
  const __nv_bfloat16 b = __float2bfloat16_rn(v);
  unsigned char* w = reinterpret_cast<unsigned char*>(wbf);
  auto put = [&](int base, int r, int k, int K) {
    *reinterpret_cast<__nv_bfloat16*>(w + 2 * base + umma::kmajor_offset(r, k, K)) = b;
  };
  if (i < OFF_B1) {
    put(BF_W1F, i / NF, i % NF, NF);
  } else if (i >= OFF_W2 && i < OFF_B2) {
    const int o = (i - OFF_W2) / NH, in = (i - OFF_W2) % NH;   // W[o][in]
    put(BF_W2F, o, in, NH);
    put(BF_W2B, in, o, NH);
  } else if (i >= OFF_W3 && i < OFF_B3) {
    const int o = (i - OFF_W3) / NH, in = (i - OFF_W3) % NH;
    put(BF_W3F, o, in, NH);
    put(BF_W3B, in, o, NH);
  }
}

// Adam on the FP32 master weights and their BF16 copies; clears the gradient.
// bc1 = 1 - beta1^step, bc2 = 1 - beta2^step.
__global__ void k_adam(float* prm, float* grad, float* m, float* v, __nv_bfloat16* wbf, float lr, float b1, float b2,
                       float eps, float bc1, float bc2) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NPARAM) return;
  float g = grad[i];
  float mi = b1 * m[i] + (1.f - b1) * g;
  float vi = b2 * v[i] + (1.f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  const float p = prm[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  prm[i] = p;
  grad[i] = 0.f;
  pack_param(i, p, wbf);
}

__global__ void k_pack_bf16(const float* __restrict__ prm, __nv_bfloat16* wbf) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NPARAM) pack_param(i, prm[i], wbf);
}

}  // namespace mlp
}  // namespace m2cg

using namespace m2cg;
using namespace m2cg::mlp;

struct m2cg_mlp {
  cudaStream_t stream = nullptr;
  int nsm = 0;
  float* prm = nullptr;  // FP32 master weights
  float* grad = nullptr;
  float* adam_m = nullptr;
  float* adam_v = nullptr;
  __nv_bfloat16* wbf = nullptr;
  float* loss = nullptr;
  int* err = nullptr;
  int64_t step = 0;
  // training set on the device
  int64_t n_data = 0;
  __nv_bfloat16* X = nullptr;
  float* y = nullptr;
  int32_t* perm = nullptr;         // two epochs' permutations of the rows
  // training: the next epoch's permutation is copied beside the current epoch
  cudaStream_t copies = nullptr;
  cudaEvent_t copied = nullptr;            // the last permutation has arrived
  cudaEvent_t used[2] = {nullptr, nullptr};  // the epoch that read perm + k n is done
  float* epoch_loss = nullptr;
  int epoch_cap = 0;
  // m2cg_mlp_predict's buffers, kept between calls up to WS_KEEP bytes (one
  // call at a time holds them): six allocations and releases a call were 0.4 of
  // 1.0 ms for 262,144 rows
  std::mutex ws_lock;
  void* ws = nullptr;
  size_t ws_bytes = 0;
};
constexpr size_t WS_KEEP = size_t(256) << 20;

namespace {
m2cg_status mlp_check(m2cg_mlp* m) {
  int herr = 0;
  MCK(cudaMemcpyAsync(&herr, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  if (herr) {
    m2cg_set_error("MLP kernel: tensor-core completion wait timed out");
    return M2CG_ERR_CUDA;
  }
  return M2CG_OK;
}
cudaError_t mlp_set_smem() {
  static bool done = false;
  if (done) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TRAIN);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_FWD);
  done = (e == cudaSuccess);
  return e;
}
}  // namespace

extern "C" {

m2cg_status m2cg_mlp_create(uint64_t seed, m2cg_mlp** out) {
  if (!out) { m2cg_set_error("null argument"); return M2CG_ERR_INVALID_ARG; }
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { m2cg_set_error("no CUDA device"); return M2CG_ERR_NO_DEVICE; }
  m2cg_mlp* m = new m2cg_mlp();
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&m->nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithFlags(&m->copies, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&m->copied, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&m->used[0], cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&m->used[1], cudaEventDisableTiming) != cudaSuccess ||
      cudaMalloc(&m->prm, NPARAM * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->grad, NPARAM * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->adam_m, NPARAM * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->adam_v, NPARAM * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&m->wbf, NBF * sizeof(__nv_bfloat16)) != cudaSuccess ||
      cudaMalloc(&m->loss, sizeof(float)) != cudaSuccess || cudaMalloc(&m->err, sizeof(int)) != cudaSuccess ||
      mlp_set_smem() != cudaSuccess) {
    m2cg_set_error("MLP allocation failed: %s", cudaGetErrorString(cudaGetLastError()));
    m2cg_mlp_destroy(m);
    return M2CG_ERR_CUDA;
  }
  // He-uniform initial weights for the SiLU layers, zero biases
  std::vector<float> h(NPARAM, 0.f);
  std::mt19937_64 rng(seed);
  auto fill = [&](int off, int fan_out, int fan_in) {
    float a = std::sqrt(6.0f / (float)fan_in);
    std::uniform_real_distribution<float> u(-a, a);
    for (int i = 0; i < fan_out * fan_in; i++) h[off + i] = u(rng);
  };
  fill(OFF_W1, NH, NF);
  for (int o = 0; o < NH; o++)
    for (int k = 12; k < NF; k++) h[OFF_W1 + o * NF + k] = 0.f;  // 12 of the 16 inputs are used
  fill(OFF_W2, NH, NH);
  fill(OFF_W3, NH, NH);
  fill(OFF_W4, 1, NH);
  for (int i = 0; i < NH; i++) h[OFF_W4 + i] *= 0.5f;
  m2cg_status st = m2cg_mlp_set_params(m, h.data());
  if (st != M2CG_OK) { m2cg_mlp_destroy(m); return st; }
  *out = m;
  return M2CG_OK;
}

void m2cg_mlp_destroy(m2cg_mlp* m) {
  if (!m) return;
  if (m->stream) cudaStreamSynchronize(m->stream);
  for (void* p : {(void*)m->prm, (void*)m->grad, (void*)m->adam_m, (void*)m->adam_v, (void*)m->wbf, (void*)m->loss,
                  (void*)m->err, (void*)m->X, (void*)m->y, (void*)m->perm, (void*)m->epoch_loss, m->ws})
    if (p) cudaFree(p);
  for (cudaEvent_t e : {m->copied, m->used[0], m->used[1]})
    if (e) cudaEventDestroy(e);
  if (m->copies) cudaStreamDestroy(m->copies);
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
}

m2cg_status m2cg_mlp_set_params(m2cg_mlp* m, const float* params) {
  if (!m || !params) { m2cg_set_error("null argument"); return M2CG_ERR_INVALID_ARG; }
  MCK(cudaMemcpyAsync(m->prm, params, NPARAM * sizeof(float), cudaMemcpyHostToDevice, m->stream));
  MCK(cudaMemsetAsync(m->grad, 0, NPARAM * sizeof(float), m->stream));
  MCK(cudaMemsetAsync(m->adam_m, 0, NPARAM * sizeof(float), m->stream));
  MCK(cudaMemsetAsync(m->adam_v, 0, NPARAM * sizeof(float), m->stream));
  MCK(cudaMemsetAsync(m->err, 0, sizeof(int), m->stream));
  k_pack_bf16<<<(NPARAM + 255) / 256, 256, 0, m->stream>>>(m->prm, m->wbf);
  MCK(cudaGetLastError());
  m->step = 0;
  MCK(cudaStreamSynchronize(m->stream));
  return M2CG_OK;
}

m2cg_status m2cg_mlp_adam_step(m2cg_mlp* m, const float* grad, float lr) {
  if (!m || !grad || !(lr > 0.f)) { m2cg_set_error("null argument or non-positive rate"); return M2CG_ERR_INVALID_ARG; }
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;   // as m2cg_mlp_train
  MCK(cudaMemcpyAsync(m->grad, grad, NPARAM * sizeof(float), cudaMemcpyHostToDevice, m->stream));
  m->step++;
  const float bc1 = 1.f - std::pow(b1, (float)m->step), bc2 = 1.f - std::pow(b2, (float)m->step);
  k_adam<<<(NPARAM + 127) / 128, 128, 0, m->stream>>>(m->prm, m->grad, m->adam_m, m->adam_v, m->wbf, lr, b1, b2, eps,
                                                      bc1, bc2);
  MCK(cudaGetLastError());
  MCK(cudaStreamSynchronize(m->stream));
  return M2CG_OK;
}

m2cg_status m2cg_mlp_get_params(m2cg_mlp* m, float* params) {
  if (!m || !params) { m2cg_set_error("null argument"); return M2CG_ERR_INVALID_ARG; }
  MCK(cudaMemcpyAsync(params, m->prm, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  return M2CG_OK;
}

m2cg_status m2cg_mlp_features(int64_t n, const double* W, const double* eos, const double* pstar, float* X,
                              float* pref, float* t) {
  if (n < 0 || !W || !eos || !X) { m2cg_set_error("null argument"); return M2CG_ERR_INVALID_ARG; }
  if (n == 0) return M2CG_OK;
  double *dW, *dE, *dp = nullptr;
  __nv_bfloat16* dX;
  float *dt = nullptr, *dref;
  MCK(cudaMalloc(&dW, n * 6 * sizeof(double)));
  MCK(cudaMalloc(&dE, n * 10 * sizeof(double)));
  MCK(cudaMalloc(&dX, n * NF * sizeof(__nv_bfloat16)));
  MCK(cudaMalloc(&dref, n * sizeof(float)));
  MCK(cudaMemcpy(dW, W, n * 6 * sizeof(double), cudaMemcpyHostToDevice));
  MCK(cudaMemcpy(dE, eos, n * 10 * sizeof(double), cudaMemcpyHostToDevice));
  if (pstar && t) {
    MCK(cudaMalloc(&dp, n * sizeof(double)));
    MCK(cudaMalloc(&dt, n * sizeof(float)));
    MCK(cudaMemcpy(dp, pstar, n * sizeof(double), cudaMemcpyHostToDevice));
  }
  k_features<<<(unsigned)((n + 255) / 256), 256>>>(n, dW, dE, dp, dX, dref, dt);
  MCK(cudaGetLastError());
  std::vector<__nv_bfloat16> h(n * NF);
  MCK(cudaMemcpy(h.data(), dX, n * NF * sizeof(__nv_bfloat16), cudaMemcpyDeviceToHost));
  for (int64_t i = 0; i < n * NF; i++) X[i] = __bfloat162float(h[i]);
  if (dt) MCK(cudaMemcpy(t, dt, n * sizeof(float), cudaMemcpyDeviceToHost));
  if (pref) MCK(cudaMemcpy(pref, dref, n * sizeof(float), cudaMemcpyDeviceToHost));
  cudaFree(dW); cudaFree(dE); cudaFree(dX); cudaFree(dref);
  if (dp) cudaFree(dp);
  if (dt) cudaFree(dt);
  return M2CG_OK;
}

m2cg_status m2cg_mlp_set_data(m2cg_mlp* m, int64_t n, const double* W, const double* eos, const double* pstar) {
  if (!m || n <= 0 || !W || !eos || !pstar) { m2cg_set_error("null argument or empty set"); return M2CG_ERR_INVALID_ARG; }
  if (n > (int64_t)INT32_MAX) { m2cg_set_error("training set too large"); return M2CG_ERR_CAPACITY; }
  for (void* p : {(void*)m->X, (void*)m->y, (void*)m->perm}) if (p) cudaFree(p);
  m->X = nullptr; m->y = nullptr; m->perm = nullptr;
  double *dW, *dE, *dp;
  MCK(cudaMalloc(&m->X, n * NF * sizeof(__nv_bfloat16)));
  MCK(cudaMalloc(&m->y, n * sizeof(float)));
  MCK(cudaMalloc(&m->perm, 2 * n * sizeof(int32_t)));
  MCK(cudaMalloc(&dW, n * 6 * sizeof(double)));
  MCK(cudaMalloc(&dE, n * 10 * sizeof(double)));
  MCK(cudaMalloc(&dp, n * sizeof(double)));
  MCK(cudaMemcpyAsync(dW, W, n * 6 * sizeof(double), cudaMemcpyHostToDevice, m->stream));
  MCK(cudaMemcpyAsync(dE, eos, n * 10 * sizeof(double), cudaMemcpyHostToDevice, m->stream));
  MCK(cudaMemcpyAsync(dp, pstar, n * sizeof(double), cudaMemcpyHostToDevice, m->stream));
  k_features<<<(unsigned)((n + 255) / 256), 256, 0, m->stream>>>(n, dW, dE, dp, m->X, nullptr, m->y);
  MCK(cudaGetLastError());
  MCK(cudaStreamSynchronize(m->stream));
  cudaFree(dW); cudaFree(dE); cudaFree(dp);
  m->n_data = n;
  return M2CG_OK;
}

m2cg_status m2cg_mlp_train(m2cg_mlp* m, int32_t epochs, int32_t batch, float lr, uint64_t seed, float* loss_per_epoch,
                           float* ms) {
  if (!m || epochs < 0 || batch < 1 || !(lr > 0.f)) { m2cg_set_error("bad training arguments"); return M2CG_ERR_INVALID_ARG; }
  if (m->n_data == 0) { m2cg_set_error("no training data (m2cg_mlp_set_data)"); return M2CG_ERR_INVALID_ARG; }
  const int64_t n = m->n_data;
  if (batch > n) batch = (int32_t)n;
  if (epochs > m->epoch_cap) {
    if (m->epoch_loss) cudaFree(m->epoch_loss);
    m->epoch_loss = nullptr;
    m->epoch_cap = 0;
    MCK(cudaMalloc(&m->epoch_loss, epochs * sizeof(float)));
    m->epoch_cap = epochs;
  }
  std::vector<int32_t> perm(n);
  for (int64_t i = 0; i < n; i++) perm[i] = (int32_t)i;
  std::mt19937_64 rng(seed);
  cudaEvent_t e0, e1;
  MCK(cudaEventCreate(&e0));
  MCK(cudaEventCreate(&e1));
  MCK(cudaEventRecord(e0, m->stream));
  if (epochs > 0) MCK(cudaMemsetAsync(m->epoch_loss, 0, epochs * sizeof(float), m->stream));
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  // The host shuffles an epoch's rows (0.35 ms for 131,072) while the device
  // works through the epoch before, from the other half of perm; the losses are
  // read once, after the last epoch (4 epochs of 131,072 rows 1.84 -> 1.38 ms).
  for (int ep = 0; ep < epochs; ep++) {
    // cosine decay from lr to lr / 20 over the epochs
    const float lr_ep = lr * (0.05f + 0.95f * 0.5f * (1.f + std::cos(3.14159265f * (float)ep / (float)epochs)));
    if (ep > 0) MCK(cudaEventSynchronize(m->copied));   // the last permutation has left perm
    std::shuffle(perm.begin(), perm.end(), rng);
    int32_t* dperm = m->perm + (ep & 1) * n;
    if (ep > 1) MCK(cudaStreamWaitEvent(m->copies, m->used[ep & 1], 0));
    MCK(cudaMemcpyAsync(dperm, perm.data(), n * sizeof(int32_t), cudaMemcpyHostToDevice, m->copies));
    MCK(cudaEventRecord(m->copied, m->copies));
    MCK(cudaStreamWaitEvent(m->stream, m->copied, 0));
    for (int64_t b0 = 0; b0 + batch <= n; b0 += batch) {  // whole batches only
      k_train<<<(unsigned)((batch + TILE - 1) / TILE), NTHR, SMEM_TRAIN, m->stream>>>(
          batch, dperm + b0, m->X, m->y, m->wbf, m->prm, m->grad, m->epoch_loss + ep, m->err);
      m->step++;
      float bc1 = 1.f - std::pow(b1, (float)m->step), bc2 = 1.f - std::pow(b2, (float)m->step);
      k_adam<<<(NPARAM + 127) / 128, 128, 0, m->stream>>>(m->prm, m->grad, m->adam_m, m->adam_v, m->wbf, lr_ep, b1, b2,
                                                          eps, bc1, bc2);
    }
    MCK(cudaGetLastError());
    MCK(cudaEventRecord(m->used[ep & 1], m->stream));
  }
  MCK(cudaEventRecord(e1, m->stream));
  if (loss_per_epoch && epochs > 0)
    MCK(cudaMemcpyAsync(loss_per_epoch, m->epoch_loss, epochs * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  if (loss_per_epoch)
    for (int ep = 0; ep < epochs; ep++) loss_per_epoch[ep] /= (float)((n / batch) * batch);
  if (ms) MCK(cudaEventElapsedTime(ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return mlp_check(m);
}

m2cg_status m2cg_mlp_grad(m2cg_mlp* m, int64_t n, const float* X, const float* t, float* grad, float* loss) {
  if (!m || n <= 0 || !X || !t || !grad) { m2cg_set_error("null argument"); return M2CG_ERR_INVALID_ARG; }
  std::vector<__nv_bfloat16> h(n * NF);
  for (int64_t i = 0; i < n * NF; i++) h[i] = __float2bfloat16_rn(X[i]);
  __nv_bfloat16* dX;
  float* dt;
  MCK(cudaMalloc(&dX, n * NF * sizeof(__nv_bfloat16)));
  MCK(cudaMalloc(&dt, n * sizeof(float)));
  MCK(cudaMemcpyAsync(dX, h.data(), n * NF * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice, m->stream));
  MCK(cudaMemcpyAsync(dt, t, n * sizeof(float), cudaMemcpyHostToDevice, m->stream));
  MCK(cudaMemsetAsync(m->grad, 0, NPARAM * sizeof(float), m->stream));
  MCK(cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream));
  k_train<<<(unsigned)((n + TILE - 1) / TILE), NTHR, SMEM_TRAIN, m->stream>>>(n, nullptr, dX, dt, m->wbf, m->prm,
                                                                              m->grad, m->loss, m->err);
  MCK(cudaGetLastError());
  MCK(cudaMemcpyAsync(grad, m->grad, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  if (loss) MCK(cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaMemsetAsync(m->grad, 0, NPARAM * sizeof(float), m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  cudaFree(dX);
  cudaFree(dt);
  if (loss) *loss /= (float)n;
  return mlp_check(m);
}

m2cg_status m2cg_mlp_forward(m2cg_mlp* m, int64_t n, const float* X, float* t) {
  if (!m || n < 0 || !X || !t) { m2cg_set_error("null argument"); return M2CG_ERR_INVALID_ARG; }
  if (n == 0) return M2CG_OK;
  std::vector<__nv_bfloat16> h(n * NF);
  for (int64_t i = 0; i < n * NF; i++) h[i] = __float2bfloat16_rn(X[i]);
  __nv_bfloat16* dX;
  float* dt;
  MCK(cudaMalloc(&dX, n * NF * sizeof(__nv_bfloat16)));
  MCK(cudaMalloc(&dt, n * sizeof(float)));
  MCK(cudaMemcpyAsync(dX, h.data(), n * NF * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice, m->stream));
  int64_t ntiles = (n + TILE - 1) / TILE;
  int grid = (int)std::min<int64_t>(ntiles, 2 * m->nsm);
  k_forward<<<grid, NTHR, SMEM_FWD, m->stream>>>(n, nullptr, dX, m->wbf, m->prm, dt, m->err, nullptr);
  MCK(cudaGetLastError());
  MCK(cudaMemcpyAsync(t, dt, n * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  cudaFree(dX);
  cudaFree(dt);
  return mlp_check(m);
}

m2cg_status m2cg_mlp_predict(m2cg_mlp* m, int64_t n, const double* W, const double* eos, double* p_pred,
                             float* kernel_ms) {
  if (!m || n < 0 || !W || !eos || !p_pred) { m2cg_set_error("null argument"); return M2CG_ERR_INVALID_ARG; }
  if (n == 0) return M2CG_OK;
  // per row: W, eos and p* (17 doubles), the network input (32 bytes), output and p_ref
  const size_t bytes = (size_t)n * (17 * sizeof(double) + NF * sizeof(__nv_bfloat16) + 2 * sizeof(float));
  std::lock_guard<std::mutex> lock(m->ws_lock);
  if (bytes > m->ws_bytes) {
    if (m->ws) cudaFree(m->ws);
    m->ws = nullptr;
    m->ws_bytes = 0;
    MCK(cudaMalloc(&m->ws, bytes));
    m->ws_bytes = bytes;
  }
  __nv_bfloat16* dX = (__nv_bfloat16*)m->ws;   // first: its rows are read in 16-byte words
  double *dW = (double*)(dX + n * NF), *dE = dW + 6 * n, *dp = dE + 10 * n;
  float *dt = (float*)(dp + n), *dref = dt + n;
  MCK(cudaMemcpyAsync(dW, W, n * 6 * sizeof(double), cudaMemcpyHostToDevice, m->stream));
  MCK(cudaMemcpyAsync(dE, eos, n * 10 * sizeof(double), cudaMemcpyHostToDevice, m->stream));
  cudaEvent_t e0, e1;
  MCK(cudaEventCreate(&e0));
  MCK(cudaEventCreate(&e1));
  MCK(cudaEventRecord(e0, m->stream));
  k_features<<<(unsigned)((n + 255) / 256), 256, 0, m->stream>>>(n, dW, dE, nullptr, dX, dref, nullptr);
  int64_t ntiles = (n + TILE - 1) / TILE;
  int grid = (int)std::min<int64_t>(ntiles, 2 * m->nsm);
  k_forward<<<grid, NTHR, SMEM_FWD, m->stream>>>(n, nullptr, dX, m->wbf, m->prm, dt, m->err, nullptr);
  k_to_pressure<<<(unsigned)std::min<int64_t>((n + 255) / 256, 65535), 256, 0, m->stream>>>(n, dt, dref, dp,
                                                                                              nullptr, nullptr, nullptr);
  MCK(cudaEventRecord(e1, m->stream));
  MCK(cudaGetLastError());
  MCK(cudaMemcpyAsync(p_pred, dp, n * sizeof(double), cudaMemcpyDeviceToHost, m->stream));
  MCK(cudaStreamSynchronize(m->stream));
  if (kernel_ms) MCK(cudaEventElapsedTime(kernel_ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (m->ws_bytes > WS_KEEP) {
    cudaFree(m->ws);
    m->ws = nullptr;
    m->ws_bytes = 0;
  }
  return mlp_check(m);
}

}  // extern "C"

// ---- use inside the finite-volume step (m2cg_api.cu) -----------------------------
namespace m2cg {
// Features of the interface faces, network, starting pressures (float) for
// the interface solve; all device-side, sized by the interface list capacity.
void mlp_warm_faces(m2cg_mlp* m, cudaStream_t s, int nsm, const Params& P, const StateSet& S, const int32_t* id,
                    const IfaceList& L, __nv_bfloat16* X, float* t, float* pref, float* warm, const DevScalars* sc) {
  k_features_faces<<<nsm * 4, 128, 0, s>>>(P, S, id, L, X, pref, sc);
  int64_t ntiles = (L.cap + TILE - 1) / TILE;
  int grid = (int)std::min<int64_t>(ntiles, 2 * nsm);
  k_forward<<<grid, NTHR, SMEM_FWD, s>>>(L.cap, L.count, X, m->wbf, m->prm, t, m->err, sc);
  k_to_pressure<<<nsm * 4, 128, 0, s>>>(L.cap, t, pref, nullptr, warm, sc, L.count);
}
cudaError_t mlp_prepare() { return mlp_set_smem(); }
}  // namespace m2cg
