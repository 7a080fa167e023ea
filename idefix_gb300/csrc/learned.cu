// Learned interface-state correction (see learned.cuh): the trainer around
// the training kernels (train_tile.cuh), the coarsening of fine snapshots and
// the learned sweep of the ORDER 5 solver (network inference fused with the
// reconstruction, the Riemann solve and the flux difference), with their C
// ABI.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "../../include/idefix_gb300.h"
#include "engine.hpp"
#include "learned.cuh"
#include "train_tile.cuh"
#include "umma.cuh"

using namespace idfx;
using namespace idfx::learn;

namespace {

// ---------------------------------------------------------------------------
// Coarsening of a fine snapshot (ghosted reference layout, 3-D, periodic):
// conserved averages over r^3 cells, face fields over r^2 faces, cell field
// from the coarse faces, ConsToPrim; and the face targets: per direction d,
// the fine primitives extrapolated to the coarse cell's two faces from the
// two fine layers next to each face (1.5 x outer layer - 0.5 x next layer;
// the outer layer alone when r = 1), averaged over the face (rotated
// variable order).
// One thread per coarse cell.  Outputs (compact, C order z, y, x):
//   prim[8][nc^3], faces[3][nc^3] (left faces), tgt[3][16][nc^3]
// ---------------------------------------------------------------------------
__global__ void k_coarsen(const double* __restrict__ Vc, const double* __restrict__ Vs, int nf, int ng, int r,
                          double gamma, double* __restrict__ prim, double* __restrict__ faces,
                          double* __restrict__ tgt) {
  const int nc = nf / r;
  const long long ncell_c = (long long)nc * nc * nc;
  const long long cid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (cid >= ncell_c) return;
  const int X = (int)(cid % nc), Y = (int)((cid / nc) % nc), Z = (int)(cid / ((long long)nc * nc));
  const int nt = nf + 2 * ng, ntv = nt + 1;
  const long long fcell = (long long)nt * nt * nt, fface = (long long)ntv * ntv * ntv;
  auto ci = [&](int k, int j, int i) { return ((long long)k * nt + j) * nt + i; };
  auto fi = [&](int k, int j, int i) { return ((long long)k * ntv + j) * ntv + i; };
  const double g1 = gamma - 1.0;
  double U[5] = {0, 0, 0, 0, 0};
  // face extrapolation weights of the fine layers along d (offset 0..r-1)
  const double wo = (r > 1) ? 1.5 : 1.0, wi = (r > 1) ? -0.5 : 0.0;
  double first[3][8], last[3][8];
  for (int d = 0; d < 3; d++)
    for (int n = 0; n < 8; n++) first[d][n] = last[d][n] = 0.0;
  for (int a = 0; a < r; a++)
    for (int b = 0; b < r; b++)
      for (int c = 0; c < r; c++) {
        const int k = ng + Z * r + a, j = ng + Y * r + b, i = ng + X * r + c;
        const long long q = ci(k, j, i);
        double V[8];
        for (int n = 0; n < 8; n++) V[n] = Vc[n * fcell + q];
        const double v2 = V[1] * V[1] + V[2] * V[2] + V[3] * V[3];
        const double b2 = V[5] * V[5] + V[6] * V[6] + V[7] * V[7];
        U[0] += V[0];
        U[1] += V[0] * V[1];
        U[2] += V[0] * V[2];
        U[3] += V[0] * V[3];
        U[4] += V[4] / g1 + 0.5 * V[0] * v2 + 0.5 * b2;
        const int off[3] = {c, b, a};
        for (int d = 0; d < 3; d++) {
          const double w0 = (off[d] == 0) ? wo : ((off[d] == 1 && r > 1) ? wi : 0.0);
          const double w1 = (off[d] == r - 1) ? wo : ((off[d] == r - 2 && r > 1) ? wi : 0.0);
          if (w0 != 0.0)
            for (int n = 0; n < 8; n++) first[d][n] += w0 * V[n];
          if (w1 != 0.0)
            for (int n = 0; n < 8; n++) last[d][n] += w1 * V[n];
        }
      }
  const double inv3 = 1.0 / ((double)r * r * r), inv2 = 1.0 / ((double)r * r);
  for (int n = 0; n < 5; n++) U[n] *= inv3;
  double Bf[3][2];
  for (int d = 0; d < 3; d++) {
    const double* vs = Vs + d * fface;
    for (int side = 0; side < 2; side++) {
      double s = 0.0;
      for (int a = 0; a < r; a++)
        for (int b = 0; b < r; b++) {
          int k, j, i;
          if (d == 0) {
            i = ng + (X + side) * r; j = ng + Y * r + b; k = ng + Z * r + a;
          } else if (d == 1) {
            j = ng + (Y + side) * r; i = ng + X * r + b; k = ng + Z * r + a;
          } else {
            k = ng + (Z + side) * r; i = ng + X * r + b; j = ng + Y * r + a;
          }
          s += vs[fi(k, j, i)];
        }
      Bf[d][side] = s * inv2;
    }
    faces[d * ncell_c + cid] = Bf[d][0];
  }
  double P[8];
  P[0] = U[0];
  for (int d = 0; d < 3; d++) P[1 + d] = U[1 + d] / U[0];
  for (int d = 0; d < 3; d++) P[5 + d] = 0.5 * (Bf[d][0] + Bf[d][1]);
  P[4] = g1 * (U[4] - 0.5 * U[0] * (P[1] * P[1] + P[2] * P[2] + P[3] * P[3]) -
               0.5 * (P[5] * P[5] + P[6] * P[6] + P[7] * P[7]));
  for (int n = 0; n < 8; n++) prim[n * ncell_c + cid] = P[n];
  for (int d = 0; d < 3; d++)
    for (int rv = 0; rv < 8; rv++) {
      const int sv = rot_var(rv, d);
      tgt[((long long)d * 16 + rv) * ncell_c + cid] = first[d][sv] * inv2;
      tgt[((long long)d * 16 + 8 + rv) * ncell_c + cid] = last[d][sv] * inv2;
    }
}

// ---------------------------------------------------------------------------
// Learned sweep (ORDER 5): reconstruction with the network's correction,
// Riemann solve and flux difference of one direction in one kernel, over
// tiles of 128 cells laid along the sweep's pencils (lines of cells along
// DIR: the active cells plus one ghost cell at each end, for every column
// of the other two directions including the CT extension).  Per tile:
//   1. stencil features of the 128 cells (BF16, canonical K-major layout);
//   2. the three layers on the 5th-generation tensor cores - one thread
//      issues tcgen05.mma over the shared-memory operands, the FP32
//      accumulators live in tensor memory, the epilogues (bias, SiLU) read
//      them back with tcgen05.ld and write the next layer's operand;
//   3. each cell's PLM (van Leer) states plus the correction, or the plain
//      PLM states where the stencil is outside the trained feature range or
//      a corrected density / pressure is not positive (the cell's two faces
//      together), kept in shared memory;
//   4. the HLLD solve of every face between two cells of the tile, its EMF
//      outputs, and the flux difference of every cell with both faces in the
//      tile (the march's expressions, so that with a zero correction the
//      sweep is bit-identical to the plain PLM march).
// Pencils of up to 128 cells are packed whole into a tile; longer pencils
// are cut into segments of 128 cells that overlap by two (the face between
// them is solved by both, with the same result).  Persistent CTAs of 256
// threads, the BF16 weights resident in shared memory.  With states != null
// the kernel writes the face states ([3][16][ncell]: direction, face
// (minus / plus) x variable) and stops before the Riemann solves.
// ---------------------------------------------------------------------------
constexpr int LT = 128;  // cells (rows) per tile
constexpr size_t LS_W1 = 0;                                  // W1: N 128 x K 224
constexpr size_t LS_W2 = LS_W1 + (size_t)NH * K1 * 2;        // W2: 128 x 128
constexpr size_t LS_W3 = LS_W2 + (size_t)NH * NH * 2;        // W3: 16 x 128
constexpr size_t LS_X = LS_W3 + (size_t)NOUT * NH * 2;       // features 128 x 224 (reused)
constexpr size_t LS_H = LS_X + (size_t)LT * K1 * 2;          // layer-1 output 128 x 128
constexpr size_t LS_B = LS_H + (size_t)LT * NH * 2;          // biases
constexpr size_t LS_R = LS_B + (size_t)(2 * NH + NOUT) * 4;  // trained range
constexpr size_t LS_F = LS_R + (size_t)2 * NIN * 4;          // per-row fallback flags
constexpr size_t LS_M = LS_F + (size_t)LT * 4;               // counter, mbarrier, TMEM slot
constexpr size_t SM_LEARN = LS_M + 32;
// inside the feature region once the network is done with it
constexpr size_t LX_Y = 0;                                   // outputs 128 x 16 FP32
constexpr size_t LX_S = LX_Y + (size_t)LT * NOUT * 4;        // face states 128 x 2 x 8 FP64
constexpr size_t LX_FA = LX_S + (size_t)LT * 16 * 8;         // flux x area 128 x 5 FP64
constexpr size_t LX_CM = LX_FA + (size_t)LT * 5 * 8;         // wave speed 128 FP64
static_assert(LX_CM + (size_t)LT * 8 <= (size_t)LT * K1 * 2, "tile outputs exceed the feature region");
static_assert(LS_X % 128 == 0 && LS_H % 128 == 0 && LS_W2 % 128 == 0 && LS_W3 % 128 == 0, "operand alignment");
static_assert(SM_LEARN <= 227 * 1024, "learned sweep does not fit in shared memory");

static_assert(LS_W2 - LS_W1 == (size_t)(PW2 - PW1) * 2 && LS_W3 - LS_W1 == (size_t)(PW3 - PW1) * 2 &&
                  LS_X - LS_W1 == (size_t)NPACK * 2,
              "the packed weights as they lie");

struct LearnedDev {
  const __nv_bfloat16* Wp;   // packed weights
  const float* w;            // packed FP32 parameters (biases)
  const float* fmin;         // [NIN] trained feature range, or null
  const float* fmax;
};

// tiling of one direction's pencils into tiles of LT cells
struct LTiles {
  int L;              // cells per pencil: n[DIR] + 2
  int per_tile;       // pencils per tile when L <= LT, else 0
  int nseg;           // segments of LT cells per pencil when L > LT
  int nA;             // pencils along the first transverse direction (with the CT extension)
  long long npencil;  // pencils
  long long ntiles;
};

__host__ inline LTiles make_tiles(const Geo& g, int dir) {
  const int A = (dir == 0) ? 1 : 0, B = (dir == 2) ? 1 : 2;
  LTiles t{};
  t.L = g.n[dir] + 2;
  t.nA = g.n[A] + 2 * g.ext;
  t.npencil = (long long)t.nA * (g.n[B] + 2 * g.ext);
  if (t.L <= LT) {
    t.per_tile = LT / t.L;
    t.nseg = 1;
    t.ntiles = (t.npencil + t.per_tile - 1) / t.per_tile;
  } else {
    t.per_tile = 0;
    t.nseg = (t.L - 2 + (LT - 2) - 1) / (LT - 2);
    t.ntiles = t.npencil * t.nseg;
  }
  return t;
}

// element (r, k) of a BF16 operand tile with K columns
__device__ __forceinline__ void put_bf16(unsigned char* base, int r, int k, int K, float v) {
  reinterpret_cast<__nv_bfloat16*>(base)[umma::kmajor_offset(r, k, K) / 2] = __float2bfloat16(v);
}

template <int DIR>
__global__ void __launch_bounds__(256, 1) k_learned_sweep(Geo g, Fields f, LearnedDev L, const Ctl* ctl, LTiles T,
                                                          int invdt, int last_dir, double* __restrict__ states,
                                                          unsigned long long* __restrict__ counters) {
  if (ctl->done) return;
  constexpr int A = (DIR == 0) ? 1 : 0, B = (DIR == 2) ? 1 : 2;
  using v = Var<3>;
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* W1s = sm + LS_W1;
  unsigned char* W2s = sm + LS_W2;
  unsigned char* W3s = sm + LS_W3;
  unsigned char* Xs = sm + LS_X;
  unsigned char* Hs = sm + LS_H;
  float* bs = reinterpret_cast<float*>(sm + LS_B);
  float* rmin = reinterpret_cast<float*>(sm + LS_R);
  float* rmax = rmin + NIN;
  int* flag = reinterpret_cast<int*>(sm + LS_F);
  int* nfall = reinterpret_cast<int*>(sm + LS_M);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + LS_M + 8);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + LS_M + 16);
  float* Ys = reinterpret_cast<float*>(Xs + LX_Y);
  double* FS = reinterpret_cast<double*>(Xs + LX_S);
  double* FA = reinterpret_cast<double*>(Xs + LX_FA);
  double* CM = reinterpret_cast<double*>(Xs + LX_CM);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // weights as the B operands (N x K, K-major)
  for (int e = tid; e < NPACK / 8; e += blockDim.x)
    reinterpret_cast<uint4*>(W1s)[e] = reinterpret_cast<const uint4*>(L.Wp)[e];
  for (int e = tid; e < NH; e += blockDim.x) {
    bs[e] = L.w[OB1 + e];
    bs[NH + e] = L.w[OB2 + e];
  }
  if (tid < NOUT) bs[2 * NH + tid] = L.w[OB3 + tid];
  const bool ranged = L.fmin != nullptr;
  for (int e = tid; e < NIN; e += blockDim.x) {
    rmin[e] = ranged ? L.fmin[e] : 0.f;
    rmax[e] = ranged ? L.fmax[e] : 0.f;
  }
  if (warp == 0) umma::tmem_alloc(slot, 256);  // layer 1: columns 0-127, layer 2: 128-255, layer 3: 0-15
  if (tid == 0) umma::mbar_init1(bar);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *slot;
  uint32_t phase = 0;
  bool ok = true;
  const int row = tid & (LT - 1), half = tid >> 7;
  const int a1 = (DIR + 1) % 3, a2 = (DIR + 2) % 3;
  const long long sd = g.s[DIR], s1 = g.s[a1], s2 = g.s[a2];
  const double dtdV = ctl->dtdV;
  const double areaT = g.A[DIR];
  double run_max = 0.0;  // max of InvDt over this thread's cells
  // one MMA run of a layer, then every thread waits (bounded) for it
  auto layer = [&](uint32_t d_col, const unsigned char* a, const unsigned char* b, int K, int N) {
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (tid == 0) {
      umma::mma_tile(tmem + d_col, umma::smem_addr(a), umma::smem_addr(b), K, umma::idesc_bf16_f32(LT, N), false);
      umma::mma_commit(bar);
    }
    const bool w = umma::mbar_wait_bounded(bar, phase, umma::kMmaSpin);
    phase ^= 1u;
    ok = __syncthreads_and(w) != 0;
    umma::fence_after_sync();
  };
  // hidden-layer epilogue: SiLU(acc + bias) -> BF16 operand of the next layer
  // (warp w: rows 32 (w % 4) .., columns 64 (w / 4) ..)
  auto hidden = [&](uint32_t d_col, const float* bias, unsigned char* out) {
    const int r = 32 * (warp & 3) + lane, c0 = 64 * (warp >> 2);
    for (int c = c0; c < c0 + 64; c += 16) {
      float x[16];
      umma::tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + d_col + (uint32_t)c, x);
#pragma unroll
      for (int i = 0; i < 16; i++) put_bf16(out, r, c + i, NH, silu_f(x[i] + bias[c + i]));
    }
  };
  for (long long tile = blockIdx.x; tile < T.ntiles && ok; tile += gridDim.x) {
    // ---- this thread's row: pencil, cell along DIR, segment ends --------
    long long pencil;
    int pos;
    bool valid, first, last;
    if (T.per_tile) {
      const int q = row / T.L;
      pos = row - q * T.L;
      pencil = tile * T.per_tile + q;
      valid = q < T.per_tile && pencil < T.npencil;
      first = pos == 0;
      last = pos == T.L - 1;
    } else {
      pencil = tile / T.nseg;
      pos = (int)(tile % T.nseg) * (LT - 2) + row;
      valid = pos < T.L;
      first = row == 0;
      last = row == LT - 1 || pos == T.L - 1;
    }
    if (!valid) {
      pencil = 0;
      pos = 1;
    }
    int ix[3];
    ix[DIR] = g.beg[DIR] - 1 + pos;
    ix[A] = g.beg[A] - g.ext + (int)(pencil % T.nA);
    ix[B] = g.beg[B] - g.ext + (int)(pencil / T.nA);
    const bool active_col = ix[A] >= g.beg[A] && ix[A] < g.end[A] && ix[B] >= g.beg[B] && ix[B] < g.end[B];
    const long long cc = cidx(g, ix[2], ix[1], ix[0]);
    if (tid < LT) flag[tid] = valid ? 0 : 1;
    if (tid == 0) *nfall = 0;
    __syncthreads();
    // ---- 1. stencil features (half 0: rotated variables 0-3, half 1: 4-7)
    {
      float cen[8];
#pragma unroll
      for (int rv = 0; rv < 8; rv++) cen[rv] = (float)f.Vc[rot_var(rv, DIR) * g.ncell + cc];
      const float cs = sqrtf((float)g.gamma * cen[4] / cen[0]), sb = sqrtf(cen[0]) * cs;
      int bad = 0;
      for (int q = 0; q < 4; q++) {
        const int rv = half * 4 + q;
        const double* base = f.Vc + rot_var(rv, DIR) * g.ncell + cc;
        for (int o2 = -1; o2 <= 1; o2++)
          for (int o1 = -1; o1 <= 1; o1++)
            for (int o0 = -1; o0 <= 1; o0++) {
              const float sv = valid ? (float)base[o0 * sd + o1 * s1 + o2 * s2] : 0.f;
              float x;
              if (rv == 0 || rv == 4) x = sv / cen[rv] - 1.f;
              else if (rv < 4) x = (sv - cen[rv]) / cs;
              else x = sv / sb;
              const int col = rv * 27 + (o2 + 1) * 9 + (o1 + 1) * 3 + (o0 + 1);
              if (!valid) x = 0.f;
              if (ranged && !(x >= rmin[col] && x <= rmax[col])) bad = 1;
              put_bf16(Xs, row, col, K1, x);
            }
      }
      if (half == 1)
        for (int col = NIN; col < K1; col++) put_bf16(Xs, row, col, K1, 0.f);
      if (bad) atomicOr(flag + row, 1);
    }
    // ---- 2. the network on the tensor cores -----------------------------
    layer(0, Xs, W1s, K1, NH);  // layer 1 -> TMEM columns 0-127
    if (!ok) break;
    hidden(0, bs, Hs);
    layer(NH, Hs, W2s, NH, NH);  // layer 2 -> TMEM columns 128-255
    if (!ok) break;
    hidden(NH, bs + NH, Xs);     // layer-2 output over the features
    layer(0, Xs, W3s, NH, NOUT);  // layer 3 -> TMEM columns 0-15
    if (!ok) break;
    if (warp < 4) {
      float y[16];
      umma::tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16), y);
#pragma unroll
      for (int i = 0; i < 16; i++) Ys[row * NOUT + i] = y[i] + bs[2 * NH + i];
    }
    __syncthreads();
    // ---- 3. corrected face states (thread: cell row, face = half) -------
    {
      double cen[8], vl[8], vr[8], st[8];
      const double dxd = g.dx[DIR];
#pragma unroll
      for (int sv = 0; sv < 8; sv++) {
        const double* base = f.Vc + sv * g.ncell + cc;
        double w[3];
        w[0] = valid ? base[-sd] : 1.0;
        w[1] = valid ? base[0] : 1.0;
        w[2] = valid ? base[sd] : 1.0;
        cen[sv] = w[1];
        Recon<2>::cell<double>(w, dxd, sv == 0 || sv == 4, vl[sv], vr[sv]);
      }
      const double cs = sqrt(g.gamma * cen[4] / cen[0]), sb = sqrt(cen[0]) * cs;
      const double sc[8] = {cen[0], cs, cs, cs, cen[4], sb, sb, sb};
#pragma unroll
      for (int rv = 0; rv < 8; rv++) {
        const int sv = rot_var(rv, DIR);
        const double plm = half ? vr[sv] : vl[sv];
        st[sv] = plm;
        if (rv == 5) continue;  // normal field: the face value is used
        st[sv] = plm + (double)Ys[row * NOUT + half * 8 + rv] * sc[rv];
      }
      if (!(st[0] > 0.0) || !(st[4] > 0.0)) atomicOr(flag + row, 1);
      __syncthreads();
      const bool fall = flag[row] != 0;
      if (fall) {
#pragma unroll
        for (int sv = 0; sv < 8; sv++) st[sv] = half ? vr[sv] : vl[sv];
      }
#pragma unroll
      for (int sv = 0; sv < 8; sv++) FS[(row * 2 + half) * 8 + sv] = st[sv];
      if (valid && states) {
#pragma unroll
        for (int sv = 0; sv < 8; sv++) states[((long long)DIR * 16 + half * 8 + sv) * g.ncell + cc] = st[sv];
      }
      if (valid && half == 0 && fall) atomicAdd(nfall, 1);
    }
    __syncthreads();
    if (tid == 0 && counters) {
      long long nvalid;
      if (T.per_tile) {
        const long long left = T.npencil - tile * T.per_tile;
        nvalid = (long long)T.L * (left < T.per_tile ? left : T.per_tile);
      } else {
        const long long p0 = (tile % T.nseg) * (LT - 2);
        nvalid = (T.L - p0 < LT) ? (T.L - p0) : LT;
      }
      atomicAdd(counters, (unsigned long long)nvalid);
      atomicAdd(counters + 1, (unsigned long long)*nfall);
    }
    if (states) continue;
    // ---- 4. Riemann solve of the face between this row and the next -----
    if (tid < LT && valid && !last) {
      double vL[8], vR[8];
#pragma unroll
      for (int n = 0; n < 8; n++) {
        vL[n] = FS[(row * 2 + 1) * 8 + n];        // plus-face state of this cell
        vR[n] = FS[((row + 1) * 2 + 0) * 8 + n];  // minus-face state of the next
      }
      int jx[3] = {ix[0], ix[1], ix[2]};
      jx[DIR] += 1;
      const long long cn = cidx(g, jx[2], jx[1], jx[0]);  // the face is the next cell's minus face
      const double bn = f.Vs[DIR * g.nface + fidx(g, jx[2], jx[1], jx[0])];
      vL[v::BX1 + DIR] = bn;
      vR[v::BX1 + DIR] = bn;
      RiemannOut<3, double> r;
      riemann<3, DIR, kHLLD>(g.gamma, g.rgm1, vL, vR, r);
      store_emf<3, DIR>(g, f, cn, r, vL, vR);
      if (active_col) {
#pragma unroll
        for (int n = 0; n < v::BX1; n++) FA[row * 5 + n] = r.F[n] * areaT;
        CM[row] = r.cmax;
      }
    }
    __syncthreads();
    // ---- flux difference of the cells with both faces in the tile -------
    if (tid < LT && valid && !first && !last && active_col) {
#pragma unroll
      for (int n = 0; n < v::BX1; n++) {
        const double rhs = -dtdV * (FA[row * 5 + n] - FA[(row - 1) * 5 + n]);
        f.Uc[n * g.ncell + cc] = f.Uc[n * g.ncell + cc] + rhs;
      }
      if (invdt) {
        const double prev = (invdt == 1) ? 0.0 : f.InvDt[cc];
        const double inv = prev + div_r(0.5 * (CM[row] + CM[row - 1]), Recip{g.dx[DIR], g.rdx[DIR]});
        f.InvDt[cc] = inv;
        if (inv > run_max) run_max = inv;  // NaN never compares greater
      }
    }
    __syncthreads();  // the feature region is rewritten by the next tile
  }
  if (!ok && tid == 0) report_wait_timeout(ctl);
  if (last_dir && invdt && !states) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, run_max, o);
      if (w > run_max) run_max = w;
    }
    if (lane == 0 && run_max > 0.0) atomic_max_pos((unsigned long long*)&((Ctl*)ctl)->invdt_max_bits, run_max);
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

__global__ void k_init_keys(unsigned* kmin, unsigned* kmax) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NIN) {
    kmin[i] = 0xffffffffu;
    kmax[i] = 0u;
  }
}

// ---------------------------------------------------------------------------
// Self-check of the tcgen05 building blocks (umma.cuh): one CTA of 128
// threads computes D[128][N] = A[128][K] . B[N][K]^T with BF16 operands staged
// in the canonical K-major layout, the FP32 accumulator in TMEM, and writes D
// from TMEM to global memory.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 1) k_umma_check(int N, int K, const __nv_bfloat16* __restrict__ A,
                                                       const __nv_bfloat16* __restrict__ B, float* __restrict__ D,
                                                       int* status) {
  extern __shared__ __align__(128) unsigned char sm[];
  __nv_bfloat16* As = reinterpret_cast<__nv_bfloat16*>(sm);
  __nv_bfloat16* Bs = reinterpret_cast<__nv_bfloat16*>(sm + 128 * K * 2);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + 128 * K * 2 + N * K * 2);
  uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int e = tid; e < 128 * K; e += blockDim.x)
    As[umma::kmajor_offset(e / K, e % K, K) / 2] = A[e];
  for (int e = tid; e < N * K; e += blockDim.x)
    Bs[umma::kmajor_offset(e / K, e % K, K) / 2] = B[e];
  uint32_t ncols = 32;
  while ((int)ncols < N) ncols *= 2;
  if (warp == 0) umma::tmem_alloc(slot, ncols);
  if (tid == 0) umma::mbar_init1(bar);
  umma::fence_async_smem();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t taddr = *slot;
  if (tid == 0) {
    umma::mma_tile(taddr, umma::smem_addr(As), umma::smem_addr(Bs), K, umma::idesc_bf16_f32(128, N), false);
    umma::mma_commit(bar);
  }
  const bool ok = umma::mbar_wait_bounded(bar, 0, umma::kMmaSpin);
  umma::fence_after_sync();
  if (ok) {
    const int row = 32 * warp + lane;
    for (int c = 0; c < N; c += 16) {
      float v[16];
      umma::tmem_ld16(taddr + ((uint32_t)(32 * warp) << 16) + (uint32_t)c, v);
#pragma unroll
      for (int i = 0; i < 16; i++) D[row * N + c + i] = v[i];
    }
  } else if (lane == 0) {
    atomicExch(status, 1);
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(taddr, ncols);
}

}  // namespace

// the network as the engine holds it (ORDER 5)
struct LearnedModel {
  __nv_bfloat16* Wp = nullptr;
  float* w = nullptr;
  float *fmin = nullptr, *fmax = nullptr;
  unsigned long long* counters = nullptr;
  bool ranged = false;
};

namespace idfx {

// the learned sweeps of one stage, direction after direction (the same
// InvDt modes as the march: 1 first contribution, 2 accumulate; the last
// direction folds the CFL maximum); states: face states instead (see
// k_learned_sweep)
static void launch_learned(Engine& e, int invdt, int fold_max, double* states) {
  LearnedModel* m = static_cast<LearnedModel*>(e.learned);
  LearnedDev L{m->Wp, m->w, m->ranged ? m->fmin : nullptr, m->ranged ? m->fmax : nullptr};
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  for (int d = 0; d < 3; d++) {
    if (e.only_dir >= 0 && e.only_dir != d) continue;
    const LTiles T = make_tiles(e.g, d);
    const int grid = (int)(T.ntiles < sms ? T.ntiles : sms);
    const int inv = (invdt == 0) ? 0 : (d == 0 ? invdt : 2);
    const int last = fold_max && d == 2;
    mark_begin(e, kKSweepX + d);
    if (d == 0) k_learned_sweep<0><<<grid, 256, SM_LEARN, e.stream>>>(e.g, e.f, L, e.ctl, T, inv, last, states, m->counters);
    if (d == 1) k_learned_sweep<1><<<grid, 256, SM_LEARN, e.stream>>>(e.g, e.f, L, e.ctl, T, inv, last, states, m->counters);
    if (d == 2) k_learned_sweep<2><<<grid, 256, SM_LEARN, e.stream>>>(e.g, e.f, L, e.ctl, T, inv, last, states, m->counters);
    mark_end(e);
  }
}

void launch_learned_sweeps(Engine& e, int invdt, int fold_max) { launch_learned(e, invdt, fold_max, nullptr); }

void free_learned(Engine& e) {
  LearnedModel* m = static_cast<LearnedModel*>(e.learned);
  if (!m) return;
  cudaFree(m->Wp);
  cudaFree(m->w);
  cudaFree(m->fmin);
  cudaFree(m->fmax);
  cudaFree(m->counters);
  delete m;
  e.learned = nullptr;
}

}  // namespace idfx

// trainer state
struct idfx_mlp {
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int max_batch = 0;
  long long t = 0;  // Adam steps taken
  float *w = nullptr, *m = nullptr, *v = nullptr, *g = nullptr;
  __nv_bfloat16* Wp = nullptr;  // packed BF16 weights
  Tile* tiles[2] = {nullptr, nullptr};  // assembled batches: the step's and the next one's
  float* part = nullptr;        // weight gradients of every block of a batch
  float* cols = nullptr;        // dZ1, dZ2, dY of every sample, by column
  double* ploss = nullptr;      // losses of every block
  double* loss = nullptr;
  unsigned *kmin = nullptr, *kmax = nullptr;
  int* status = nullptr;  // set by a block whose bounded wait gave up
  const float* prims = nullptr;
  const float* tgt = nullptr;
  int nsnap = 0, nc = 0;
  double gamma = 5.0 / 3.0;
  std::vector<void*> allocs;
};

namespace {

template <typename P>
bool dalloc(idfx_mlp* h, P** p, size_t n) {
  if (cudaMalloc(reinterpret_cast<void**>(p), n * sizeof(P)) != cudaSuccess) return false;
  h->allocs.push_back(*p);
  return cudaMemsetAsync(*p, 0, n * sizeof(P), h->stream) == cudaSuccess;
}

Dataset dataset(const idfx_mlp* h) { return Dataset{h->prims, h->tgt, h->nsnap, h->nc, (float)h->gamma}; }

// the blocks of a launch: those that put a batch through the network
// (compute) and those that assemble one into the trainer's tiles
TrainArgs batch_args(const idfx_mlp* h, int B) {
  TrainArgs a{};
  a.B = B;
  a.split = split_batch(B);
  a.cols = h->cols;
  a.ld = h->max_batch;
  a.Wp = h->Wp;
  a.w = h->w;
  a.status = h->status;
  a.D = dataset(h);
  return a;
}
void launch_tiles(idfx_mlp* h, const TrainArgs& a) {
  const unsigned n = (unsigned)(a.compute + (a.next ? a.split.blocks * a.split.tiles : 0));
  k_train_tile<<<n, TT, SM_TRAIN, h->stream>>>(a);
}
// samples base .. base + B - 1 of a seed into the tiles of `slot`
void launch_assemble(idfx_mlp* h, int B, unsigned long long seed, long long base, int slot, bool range) {
  TrainArgs a = batch_args(h, B);
  a.seed = seed;
  a.base = base;
  a.next = h->tiles[slot];
  a.kmin = range ? h->kmin : nullptr;
  a.kmax = range ? h->kmax : nullptr;
  launch_tiles(h, a);
}
// the blocks' gradients and losses summed, and the Adam step where adam.w is set
void launch_update(idfx_mlp* h, int B, bool grad, const AdamArgs& adam, double* loss) {
  k_train_update<<<grad ? UPDATE_BLOCKS : 1, 256, 0, h->stream>>>(grad ? h->part : nullptr, h->cols, h->max_batch,
                                                                 split_batch(B).blocks, h->g, adam, h->ploss, B, loss);
}

int sync_ok(idfx_mlp* h) {
  if (cudaGetLastError() != cudaSuccess) return IDFX_ERR_CUDA;
  if (cudaStreamSynchronize(h->stream) != cudaSuccess) return IDFX_ERR_CUDA;
  if (h->status) {  // a bounded tensor-core wait that gave up
    int st = 0;
    if (cudaMemcpy(&st, h->status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess || st) return IDFX_ERR_CUDA;
  }
  return IDFX_OK;
}

}  // namespace

extern "C" {

int idfx_gpu_set_learned(idfx_gpu* hg, const float* params, const float* fmin, const float* fmax) {
  if (!hg || !params) return IDFX_ERR_STATE;
  Engine& e = hg->e;
  if (e.g.order != IDFX_LEARNED) {
    e.err = "set_learned: the handle was not created with the learned reconstruction order";
    return IDFX_ERR_CONFIG;
  }
  if (cudaStreamSynchronize(e.stream) != cudaSuccess) return IDFX_ERR_CUDA;
  if (!e.learned) {
    LearnedModel* m = new (std::nothrow) LearnedModel();
    if (!m) return IDFX_ERR_STATE;
    e.learned = m;
    bool ok = cudaMalloc(&m->Wp, sizeof(__nv_bfloat16) * NPACK) == cudaSuccess;
    ok = ok && cudaMalloc(&m->w, sizeof(float) * NPARAM) == cudaSuccess;
    ok = ok && cudaMalloc(&m->fmin, sizeof(float) * NIN) == cudaSuccess;
    ok = ok && cudaMalloc(&m->fmax, sizeof(float) * NIN) == cudaSuccess;
    ok = ok && cudaMalloc(&m->counters, sizeof(unsigned long long) * 2) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(k_learned_sweep<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)SM_LEARN) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(k_learned_sweep<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)SM_LEARN) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(k_learned_sweep<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)SM_LEARN) == cudaSuccess;
    if (!ok) {
      free_learned(e);
      e.err = "set_learned: CUDA allocation failed";
      return IDFX_ERR_CUDA;
    }
  }
  LearnedModel* m = static_cast<LearnedModel*>(e.learned);
  m->ranged = fmin && fmax;
  bool ok = cudaMemcpyAsync(m->w, params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice, e.stream) == cudaSuccess;
  if (m->ranged) {
    ok = ok && cudaMemcpyAsync(m->fmin, fmin, sizeof(float) * NIN, cudaMemcpyHostToDevice, e.stream) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(m->fmax, fmax, sizeof(float) * NIN, cudaMemcpyHostToDevice, e.stream) == cudaSuccess;
  }
  ok = ok && cudaMemsetAsync(m->counters, 0, sizeof(unsigned long long) * 2, e.stream) == cudaSuccess;
  if (!ok) return IDFX_ERR_CUDA;
  k_pack_weights<<<(NPARAM + 255) / 256, 256, 0, e.stream>>>(m->w, m->Wp);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(e.stream) != cudaSuccess) return IDFX_ERR_CUDA;
  return IDFX_OK;
}

int idfx_gpu_learned_states(idfx_gpu* hg, double* ls) {
  if (!hg || !ls || !hg->e.learned) return IDFX_ERR_STATE;
  Engine& e = hg->e;
  if (idfx_gpu_set_boundaries(hg) != IDFX_OK) return IDFX_ERR_CUDA;
  const size_t n = (size_t)48 * e.g.ncell;
  double* tmp = nullptr;
  if (cudaMalloc(&tmp, n * sizeof(double)) != cudaSuccess) return IDFX_ERR_CUDA;
  bool ok = cudaMemsetAsync(tmp, 0, n * sizeof(double), e.stream) == cudaSuccess;
  if (ok) {
    launch_learned(e, 0, 0, tmp);
    ok = cudaGetLastError() == cudaSuccess;
  }
  ok = ok && cudaMemcpyAsync(ls, tmp, n * sizeof(double), cudaMemcpyDeviceToHost, e.stream) == cudaSuccess;
  ok = ok && cudaStreamSynchronize(e.stream) == cudaSuccess;
  cudaFree(tmp);
  return ok ? IDFX_OK : IDFX_ERR_CUDA;
}

int idfx_gpu_learned_stats(idfx_gpu* hg, long long* cells, long long* fallbacks) {
  if (!hg || !hg->e.learned) return IDFX_ERR_STATE;
  Engine& e = hg->e;
  unsigned long long c[2];
  LearnedModel* m = static_cast<LearnedModel*>(e.learned);
  if (cudaMemcpyAsync(c, m->counters, sizeof(c), cudaMemcpyDeviceToHost, e.stream) != cudaSuccess ||
      cudaStreamSynchronize(e.stream) != cudaSuccess)
    return IDFX_ERR_CUDA;
  if (cells) *cells = (long long)c[0];
  if (fallbacks) *fallbacks = (long long)c[1];
  return IDFX_OK;
}

int idfx_check_umma(int N, int K, const float* A, const float* B, float* D) {
  if (!A || !B || !D || N < 16 || N > 256 || N % 16 || K < 16 || K > 256 || K % 16) return IDFX_ERR_CONFIG;
  std::vector<__nv_bfloat16> a((size_t)128 * K), b((size_t)N * K);
  for (size_t i = 0; i < a.size(); i++) a[i] = __float2bfloat16(A[i]);
  for (size_t i = 0; i < b.size(); i++) b[i] = __float2bfloat16(B[i]);
  __nv_bfloat16 *da = nullptr, *db = nullptr;
  float* dd = nullptr;
  int* dst = nullptr;
  int st = 0;
  const size_t smem = (size_t)128 * K * 2 + (size_t)N * K * 2 + 16;
  bool ok = cudaMalloc(&da, a.size() * 2) == cudaSuccess && cudaMalloc(&db, b.size() * 2) == cudaSuccess &&
            cudaMalloc(&dd, (size_t)128 * N * 4) == cudaSuccess && cudaMalloc(&dst, sizeof(int)) == cudaSuccess;
  ok = ok && cudaMemcpy(da, a.data(), a.size() * 2, cudaMemcpyHostToDevice) == cudaSuccess;
  ok = ok && cudaMemcpy(db, b.data(), b.size() * 2, cudaMemcpyHostToDevice) == cudaSuccess;
  ok = ok && cudaMemset(dst, 0, sizeof(int)) == cudaSuccess && cudaMemset(dd, 0, (size_t)128 * N * 4) == cudaSuccess;
  ok = ok && cudaFuncSetAttribute(k_umma_check, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
                 cudaSuccess;
  if (ok) {
    k_umma_check<<<1, 128, smem>>>(N, K, da, db, dd, dst);
    ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
  }
  ok = ok && cudaMemcpy(D, dd, (size_t)128 * N * 4, cudaMemcpyDeviceToHost) == cudaSuccess;
  ok = ok && cudaMemcpy(&st, dst, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(da);
  cudaFree(db);
  cudaFree(dd);
  cudaFree(dst);
  if (!ok) return IDFX_ERR_CUDA;
  return st ? IDFX_ERR_CUDA : IDFX_OK;
}

int idfx_mlp_create(int max_batch, void* stream, idfx_mlp** out) {
  if (!out || max_batch < 1) return IDFX_ERR_STATE;
  *out = nullptr;
  idfx_mlp* h = new (std::nothrow) idfx_mlp();
  if (!h) return IDFX_ERR_STATE;
  if (stream) {
    h->stream = (cudaStream_t)stream;
  } else {
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) {
      delete h;
      return IDFX_ERR_CUDA;
    }
    h->own_stream = true;
  }
  h->max_batch = max_batch;
  // tiles of the worst batch: three chunks of 64 samples per block, two tiles
  const size_t tiles = 2 * (((size_t)max_batch + 63) / 64 / 3 + 2);
  const size_t B = (size_t)max_batch;
  bool ok = dalloc(h, &h->w, NPARAM) && dalloc(h, &h->m, NPARAM) && dalloc(h, &h->v, NPARAM) &&
            dalloc(h, &h->g, NPARAM) && dalloc(h, &h->Wp, NPACK) && dalloc(h, &h->tiles[0], tiles) && dalloc(h, &h->tiles[1], tiles) &&
            dalloc(h, &h->part, (size_t)MAX_BLOCKS * NPARAM) && dalloc(h, &h->cols, B * NBIAS) &&
            dalloc(h, &h->ploss, MAX_BLOCKS * 2) && dalloc(h, &h->loss, 2) && dalloc(h, &h->kmin, NIN) &&
            dalloc(h, &h->kmax, NIN) && dalloc(h, &h->status, 1);
  ok = ok && cudaFuncSetAttribute(k_train_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM_TRAIN) ==
                 cudaSuccess;
  if (ok) {
    k_init_keys<<<1, 256, 0, h->stream>>>(h->kmin, h->kmax);
    ok = sync_ok(h) == IDFX_OK;
  }
  if (!ok) {
    idfx_mlp_destroy(h);
    return IDFX_ERR_CUDA;
  }
  *out = h;
  return IDFX_OK;
}

int idfx_mlp_destroy(idfx_mlp* h) {
  if (!h) return IDFX_ERR_STATE;
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (void* p : h->allocs) cudaFree(p);
  if (h->own_stream) cudaStreamDestroy(h->stream);
  delete h;
  return IDFX_OK;
}

int idfx_mlp_set_params(idfx_mlp* h, const float* params) {
  if (!h || !params) return IDFX_ERR_STATE;
  if (cudaMemcpyAsync(h->w, params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice, h->stream) != cudaSuccess)
    return IDFX_ERR_CUDA;
  cudaMemsetAsync(h->m, 0, sizeof(float) * NPARAM, h->stream);
  cudaMemsetAsync(h->v, 0, sizeof(float) * NPARAM, h->stream);
  h->t = 0;
  k_pack_weights<<<(NPARAM + 255) / 256, 256, 0, h->stream>>>(h->w, h->Wp);
  return sync_ok(h);
}

int idfx_mlp_get_params(idfx_mlp* h, float* params) {
  if (!h || !params) return IDFX_ERR_STATE;
  if (cudaMemcpyAsync(params, h->w, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, h->stream) != cudaSuccess)
    return IDFX_ERR_CUDA;
  return sync_ok(h);
}

int idfx_mlp_set_dataset_device(idfx_mlp* h, const float* prims, const float* targets, int nsnap, int nc,
                                double gamma) {
  if (!h || !prims || !targets || nsnap < 1 || nc < 3) return IDFX_ERR_STATE;
  h->prims = prims;
  h->tgt = targets;
  h->nsnap = nsnap;
  h->nc = nc;
  h->gamma = gamma;
  return IDFX_OK;
}

int idfx_mlp_batch_device(idfx_mlp* h, int batch, unsigned long long seed, long long base, void* X, float* T) {
  if (!h || !h->prims || !X || !T || batch < 1) return IDFX_ERR_STATE;
  k_make_batch<<<(batch + 31) / 32, 256, 0, h->stream>>>(dataset(h), seed, base, batch,
                                                         static_cast<__nv_bfloat16*>(X), T);
  return sync_ok(h);
}

int idfx_mlp_train(idfx_mlp* h, int steps, int batch, float lr, float lr_end, unsigned long long seed,
                   float* losses) {
  if (!h || !h->prims || batch < 1 || batch > h->max_batch || steps < 0) return IDFX_ERR_STATE;
  double* dl = nullptr;
  if (cudaMalloc(&dl, sizeof(double) * 2 * (steps > 0 ? steps : 1)) != cudaSuccess) return IDFX_ERR_CUDA;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  if (steps > 0) launch_assemble(h, batch, seed, h->t * (long long)batch, 0, true);
  for (int s = 0; s < steps; s++) {
    TrainArgs a = batch_args(h, batch);
    a.compute = a.split.blocks;
    a.tiles = h->tiles[s & 1];
    a.part = h->part;
    a.loss = h->ploss;
    if (s + 1 < steps) {  // the next step's batch, meanwhile
      a.next = h->tiles[(s + 1) & 1];
      a.seed = seed;
      a.base = (h->t + s + 1) * (long long)batch;
      a.kmin = h->kmin;
      a.kmax = h->kmax;
    }
    launch_tiles(h, a);
    const double tt = (double)(h->t + s + 1);
    const float frac = steps > 1 ? (float)s / (float)(steps - 1) : 1.f;
    const float lr_s = lr_end + 0.5f * (lr - lr_end) * (1.f + cosf(3.14159265f * frac));
    launch_update(h, batch, true,
                  AdamArgs{lr_s, b1, b2, eps, (float)(1.0 - std::pow((double)b1, tt)),
                           (float)(1.0 - std::pow((double)b2, tt)), h->w, h->m, h->v, h->Wp},
                  dl + 2 * s);
  }
  h->t += steps;
  int rc = sync_ok(h);
  if (!rc && losses && steps > 0) {
    std::vector<double> hl(2 * (size_t)steps);
    if (cudaMemcpy(hl.data(), dl, sizeof(double) * 2 * steps, cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = IDFX_ERR_CUDA;
    for (int s = 0; s < steps; s++) losses[s] = (float)hl[2 * s];
  }
  cudaFree(dl);
  return rc;
}

int idfx_mlp_eval(idfx_mlp* h, int batch, unsigned long long seed, double* loss, double* loss_zero) {
  if (!h || !h->prims || batch < 1 || batch > h->max_batch) return IDFX_ERR_STATE;
  launch_assemble(h, batch, seed, 0, 0, false);
  TrainArgs a = batch_args(h, batch);
  a.compute = a.split.blocks;
  a.tiles = h->tiles[0];
  a.loss = h->ploss;
  launch_tiles(h, a);
  launch_update(h, batch, false, AdamArgs{}, h->loss);
  double hl[2];
  if (cudaMemcpyAsync(hl, h->loss, sizeof(hl), cudaMemcpyDeviceToHost, h->stream) != cudaSuccess) return IDFX_ERR_CUDA;
  const int rc = sync_ok(h);
  if (loss) *loss = hl[0];
  if (loss_zero) *loss_zero = hl[1];
  return rc;
}

int idfx_mlp_feature_range(idfx_mlp* h, float* fmin, float* fmax) {
  if (!h || !fmin || !fmax) return IDFX_ERR_STATE;
  unsigned a[NIN], b[NIN];
  cudaMemcpyAsync(a, h->kmin, sizeof(a), cudaMemcpyDeviceToHost, h->stream);
  cudaMemcpyAsync(b, h->kmax, sizeof(b), cudaMemcpyDeviceToHost, h->stream);
  const int rc = sync_ok(h);
  for (int i = 0; i < NIN; i++) {
    fmin[i] = fkey_inv(a[i]);
    fmax[i] = fkey_inv(b[i]);
  }
  return rc;
}

int idfx_mlp_grad_device(idfx_mlp* h, const void* X, const float* T, int batch, float* grad, double* loss) {
  if (!h || !X || !T || !grad || batch < 1 || batch > h->max_batch) return IDFX_ERR_STATE;
  TrainArgs a = batch_args(h, batch);
  a.compute = a.split.blocks;
  a.X = static_cast<const __nv_bfloat16*>(X);
  a.T = T;
  a.part = h->part;
  a.loss = h->ploss;
  launch_tiles(h, a);
  launch_update(h, batch, true, AdamArgs{}, h->loss);
  cudaMemcpyAsync(grad, h->g, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, h->stream);
  double hl = 0.0;
  cudaMemcpyAsync(&hl, h->loss, sizeof(double), cudaMemcpyDeviceToHost, h->stream);
  const int rc = sync_ok(h);
  if (loss) *loss = hl;
  return rc;
}

int idfx_mlp_forward_device(idfx_mlp* h, const void* X, int batch, float* Y) {
  if (!h || !X || !Y || batch < 1 || batch > h->max_batch) return IDFX_ERR_STATE;
  TrainArgs a = batch_args(h, batch);
  a.compute = a.split.blocks;
  a.X = static_cast<const __nv_bfloat16*>(X);
  a.Y = Y;
  launch_tiles(h, a);
  return sync_ok(h);
}

int idfx_learn_coarsen_device(const double* Vc, const double* Vs, int nf, int nghost, int r, double gamma,
                              double* prim, double* faces, double* targets, void* stream) {
  if (!Vc || !Vs || !prim || !faces || !targets || r < 1 || nf < r || nf % r != 0 || nghost < 1)
    return IDFX_ERR_CONFIG;
  const long long nc = nf / r;
  const long long n = nc * nc * nc;
  k_coarsen<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)stream>>>(Vc, Vs, nf, nghost, r, gamma, prim, faces,
                                                                          targets);
  if (cudaGetLastError() != cudaSuccess) return IDFX_ERR_CUDA;
  return cudaStreamSynchronize((cudaStream_t)stream) == cudaSuccess ? IDFX_OK : IDFX_ERR_CUDA;
}

}  // extern "C"
