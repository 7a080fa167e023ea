// Learned interface-state correction (see learned.cuh): the trainer around
// the training kernels (train_tile.cuh), the coarsening of fine snapshots, the
// network's corrections of a stage of the ORDER 5 solver and its sweeps (the
// cell sweep on the corrected PLM states), with their C ABI.
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
#include "learned_window.cuh"
#include "sweep_cell.cuh"
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
// Learned correction (ORDER 5): the network over every cell whose face states
// a sweep reconstructs, for the three directions in one launch; the sweeps
// (k_sweep_learned: the cell sweep of the FP64 path) add the correction
// to the PLM states.  Together in one kernel per direction, 128 of its 256
// threads solved FP64 Riemann problems while the tensor core and the other
// half waited, features were gathered from FP64 three times over, and a 32^3
// box left 2.5 tiles per multiprocessor to each of six launches a cycle.
// A tile is 128 consecutive cells of the box of those cells (x fastest):
//   1. the scaled stencil of every cell once, as BF16, [variable][neighbour][cell];
//      the three directions' inputs are permutations of it;
//   2. per direction: its input in the canonical K-major layout, the three
//      layers on the tensor cores (umma.cuh; the next layer's operand over the
//      last one's), and the sixteen outputs to Y [3][16][ncell] - the first a
//      NaN where the stencil leaves the trained range, which the sweep takes
//      as it takes a correction that leaves a density or pressure not positive.
// Persistent blocks of 512 threads (four per cell), the packed weights fetched
// by one bulk copy; a block's share is a run of (tile, direction) pairs, so
// that a small box is spread over all multiprocessors (12^3: 66 pairs of 22
// tiles) and a middling one leaves no round nearly empty (32^3: 307 tiles are
// three rounds of 152 blocks, 921 pairs seven of a third each).
// Measured (32^3, both stages of a cycle): the three fused sweeps 434 / 469 /
// 472 us; this launch 185 us (241 with whole tiles to a block and the range
// looked up by column) and the three sweeps 91 / 93 / 95 us.  Two cycles with
// their copies 3356 -> 1085 us, one cycle of 64^3 13978 -> 2650 us.
// ---------------------------------------------------------------------------
constexpr int LT = 128;   // cells of a tile
constexpr int LN = 512;   // threads
constexpr size_t LS_W = 0;                                   // packed weights
constexpr size_t LS_X = LS_W + (size_t)NPACK * 2;            // input 128 x 224, then the layers' outputs
constexpr size_t LS_F = LS_X + (size_t)LT * K1 * 2;          // scaled stencil [216][128] BF16
constexpr size_t LS_B = LS_F + (size_t)NIN * LT * 2;         // biases
constexpr size_t LS_R = LS_B + (size_t)(2 * NH + NOUT) * 4;  // trained range of a stencil element, per direction
constexpr size_t LS_O = LS_R + (size_t)3 * NIN * 8;          // cells outside it, per direction
constexpr size_t LS_M = LS_O + (size_t)3 * LT * 4;           // mbarriers, TMEM slot
constexpr size_t SM_LEARN = LS_M + 32;
static_assert(LS_X % 128 == 0 && LS_M % 8 == 0, "operand alignment");
static_assert(SM_LEARN <= 227 * 1024, "learned correction does not fit in shared memory");

struct LearnedDev {
  const __nv_bfloat16* Wp;   // packed weights
  const float* w;            // packed FP32 parameters (biases)
  const float* fmin;         // [NIN] trained feature range, or null
  const float* fmax;
};

// the cells that get a correction: lo .. lo + m - 1 in every direction
struct LBox {
  int lo[3], m[3];
  long long cells;
};
__host__ inline LBox learned_box(const Geo& g) {
  LBox b{};
  const int e = g.ext > 1 ? g.ext : 1;  // columns of the CT extension, the ghost cell at a line's ends
  b.cells = 1;
  for (int d = 0; d < 3; d++) {
    b.lo[d] = g.beg[d] - e;
    b.m[d] = g.n[d] + 2 * e;
    b.cells *= b.m[d];
  }
  return b;
}

// stencil element (solver variable * 27 + neighbour, x fastest) of feature
// column col of direction d (rotated variable, then neighbour with the sweep
// direction fastest)
__host__ __device__ constexpr int stencil_of(int d, int col) {
  const int rv = col / 27, q = col % 27;
  int o[3] = {0, 0, 0};
  o[d] = q % 3;
  o[(d + 1) % 3] = q / 3 % 3;
  o[(d + 2) % 3] = q / 9;
  return rot_var(rv, d) * 27 + o[2] * 9 + o[1] * 3 + o[0];
}
struct StencilTable {
  unsigned char at[3][K1];
};
constexpr StencilTable stencil_table() {
  StencilTable t{};
  for (int d = 0; d < 3; d++)
    for (int c = 0; c < NIN; c++) t.at[d][c] = (unsigned char)stencil_of(d, c);
  return t;
}
__constant__ StencilTable kStencil = stencil_table();
static_assert(NIN <= 256, "stencil element in a byte");

// LEAN: the cells of a window (learned_window.cuh) in its direction, the
// primitives rounded from FP64 here, the corrections at Y [16][room]
template <bool LEAN>
__global__ void __launch_bounds__(LN, 1)
    k_learned_correct(Geo g, const float* __restrict__ Vc, const double* __restrict__ Vc64, LearnedDev L, Ctl* ctl,
                      LBox box, LearnedWindow win, float* __restrict__ Y, long long room) {
  if (ctl->done) return;
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* Xs = sm + LS_X;
  __nv_bfloat16* Fs = reinterpret_cast<__nv_bfloat16*>(sm + LS_F);
  float* bs = reinterpret_cast<float*>(sm + LS_B);
  float2* range = reinterpret_cast<float2*>(sm + LS_R);
  int* out = reinterpret_cast<int*>(sm + LS_O);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + LS_M);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + LS_M + 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = 32 * (warp & 3) + lane, quarter = warp >> 2;
  const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
  if (warp == 0) umma::tmem_alloc(slot, 256);  // layer 1: columns 0-127, layer 2: 128-255, layer 3: 0-15
  if (tid == 0) {
    umma::mbar_init1(bar);
    mbar_init(bar + 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect(bar + 1, NPACK * 2);
    bulk_to_smem(sm + LS_W, L.Wp, NPACK * 2, bar + 1);
  }
  for (int e = tid; e < NH; e += LN) {
    bs[e] = L.w[OB1 + e];
    bs[NH + e] = L.w[OB2 + e];
  }
  if (tid < NOUT) bs[2 * NH + tid] = L.w[OB3 + tid];
  const bool ranged = L.fmin != nullptr;
  if (ranged) {
    for (int e = tid; e < 3 * NIN; e += LN) {
      const int d = e / NIN, c = e % NIN;
      range[3 * kStencil.at[d][c] + d] = make_float2(L.fmin[c], L.fmax[c]);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *slot;
  const uint32_t xa = umma::smem_addr(Xs), w1 = umma::smem_addr(sm + LS_W), w2 = w1 + PW2 * 2, w3 = w1 + PW3 * 2;
  uint32_t phase = 0;
  auto tensor = [&](uint32_t d_col, int K, uint32_t w, int N) -> bool {
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (tid == 0) {
      umma::mma_run(tmem + d_col, umma::along_columns(xa, K), umma::along_columns(w, K), LT, N, K);
      umma::mma_commit(bar);
    }
    const bool in = umma::mbar_wait_bounded(bar, phase, umma::kMmaSpin);
    phase ^= 1u;
    const bool ok = __syncthreads_and(in) != 0;
    umma::fence_after_sync();
    return ok;
  };
  // SiLU(acc + bias) -> BF16 operand of the next layer, in the input's place
  auto hidden = [&](uint32_t d_col, const float* bias) {
    for (int c = NH / 4 * quarter; c < NH / 4 * (quarter + 1); c += 16) {
      float x[16];
      umma::tmem_ld16(tmem + lanes + d_col + (uint32_t)c, x);
#pragma unroll
      for (int i = 0; i < 16; i++) x[i] = silu_f(x[i] + bias[c + i]);
      put8(Xs, row, c, NH, x);
      put8(Xs, row, c + 8, NH, x + 8);
    }
  };
  bool ok = __syncthreads_and(mbar_wait(bar + 1, 0u)) != 0;  // the weights
  constexpr int ND = LEAN ? 1 : 3;  // directions of a tile
  const long long cells = LEAN ? (long long)win.lines * win.per : box.cells;
  const int tiles = (int)((cells + LT - 1) / LT);
  // this block's share of all tiles' directions, in a row
  int item = (int)((long long)ND * tiles * blockIdx.x / gridDim.x);
  const int end = (int)((long long)ND * tiles * (blockIdx.x + 1) / gridDim.x);
  auto prim = [&](int v, long long c) -> float {
    if constexpr (LEAN) return d2f_rn(Vc64[v * g.ncell + c]);
    else return Vc[v * g.ncell + c];
  };
  while (item < end && ok) {
    const long long q = (long long)(item / ND) * LT + row;
    const bool valid = q < cells;
    const unsigned p = valid ? (unsigned)q : 0u;  // cells of a box fit 31 bits
    int ix[3];
    if constexpr (LEAN) {
      const int d = win.dir, a = d == 0 ? 1 : 0, b = d == 2 ? 1 : 2;
      unsigned line, pos;
      window_cell(win, p, line, pos);
      const unsigned na = (unsigned)(g.n[a] + 2 * g.ext);
      const int at[3] = {g.beg[d] - 1 + (int)pos, g.beg[a] - g.ext + (int)(line % na),
                         g.beg[b] - g.ext + (int)(line / na)};  // along d, a, b
      ix[0] = d == 0 ? at[0] : at[1];
      ix[1] = d == 0 ? at[1] : d == 1 ? at[0] : at[2];
      ix[2] = d == 2 ? at[0] : at[2];
    } else {
      ix[0] = box.lo[0] + (int)(p % (unsigned)box.m[0]);
      ix[1] = box.lo[1] + (int)(p / (unsigned)box.m[0] % (unsigned)box.m[1]);
      ix[2] = box.lo[2] + (int)(p / (unsigned)box.m[0] / (unsigned)box.m[1]);
    }
    const long long cc = cidx(g, ix[2], ix[1], ix[0]);
    for (int e = tid; e < 3 * LT; e += LN) out[e] = 0;
    __syncthreads();
    // ---- the scaled stencil, two variables per thread ------------------
    {
      const float rho = prim(0, cc), prs = prim(4, cc);
      const float cs = sqrtf((float)g.gamma * prs / rho), sb = sqrtf(rho) * cs;
      int bad = 0;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int v = 2 * quarter + k;
        const float cen = prim(v, cc);
#pragma unroll
        for (int oz = -1; oz <= 1; oz++)
#pragma unroll
          for (int oy = -1; oy <= 1; oy++)
#pragma unroll
            for (int ox = -1; ox <= 1; ox++) {
              // inside the array whatever the extension (uct_hll(d) takes a
              // column more than the stencil has around it)
              const int nx = min(max(ix[0] + ox, 0), g.nt[0] - 1), ny = min(max(ix[1] + oy, 0), g.nt[1] - 1),
                        nz = min(max(ix[2] + oz, 0), g.nt[2] - 1);
              const float s = prim(v, cidx(g, nz, ny, nx));
              float x;
              if (v == 0 || v == 4) x = s / cen - 1.f;
              else if (v < 4) x = zdiv(s - cen, cs);
              else x = zdiv(s, sb);
              const int nb = (oz + 1) * 9 + (oy + 1) * 3 + (ox + 1);
              Fs[(v * 27 + nb) * LT + row] = __float2bfloat16(valid ? x : 0.f);
              if (ranged) {
#pragma unroll
                for (int d = 0; d < 3; d++) {
                  const float2 r = range[3 * (v * 27 + nb) + d];
                  if (!(x >= r.x && x <= r.y)) bad |= 1 << d;
                }
              }
            }
      }
#pragma unroll
      for (int d = 0; d < 3; d++)
        if (bad & (1 << d)) out[d * LT + row] = 1;  // (any of the cell's threads)
    }
    __syncthreads();
    const int d0 = LEAN ? win.dir : item % 3;
    for (int d = d0; d < (LEAN ? d0 + 1 : 3) && item < end && ok; d++, item++) {
      for (int c = 8 * quarter; c < K1; c += 32) {  // this direction's input, eight columns at a time
        alignas(16) __nv_bfloat16 t[8];
#pragma unroll
        for (int i = 0; i < 8; i++)
          t[i] = c + i < NIN ? Fs[(int)kStencil.at[d][c + i] * LT + row] : __float2bfloat16(0.f);
        *reinterpret_cast<uint4*>(Xs + umma::kmajor_offset(row, c, K1)) = *reinterpret_cast<const uint4*>(t);
      }
      ok = tensor(0, K1, w1, NH);  // layer 1 -> TMEM columns 0-127
      if (!ok) break;
      hidden(0, bs);
      ok = tensor(NH, NH, w2, NH);  // layer 2 -> TMEM columns 128-255
      if (!ok) break;
      hidden(NH, bs + NH);
      ok = tensor(0, NH, w3, NOUT);  // layer 3 -> TMEM columns 0-15
      if (!ok) break;
      float y[16];
      umma::tmem_ld16(tmem + lanes, y);
      if (valid) {
#pragma unroll
        for (int o = 0; o < NOUT; o++) {
          if (o / 4 != quarter) continue;
          float z = y[o] + bs[2 * NH + o];
          if (o == 0 && out[d * LT + row]) z = __int_as_float(0x7fffffff);
          if constexpr (LEAN) Y[o * room + q] = z;
          else Y[((long long)d * NOUT + o) * g.ncell + cc] = z;
        }
      }
    }
    __syncthreads();  // the stencil and its flags are rewritten by the next tile
  }
  if (!ok && tid == 0) {
    report_wait_timeout(ctl);
    mbar_wait(bar + 1, 0u);  // no copy may land after the block has gone
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}

// the cell sweep with PLM plus the correction (sweep_cell.cuh, ORDER 5)
template <int DIR, bool WINDOW>
__global__ void __launch_bounds__(kCellThreads, cell_resident(8))
    k_sweep_learned(Geo g, Fields f, const Ctl* ctl, int invdt, int last_dir, LearnedRecon<WINDOW> lr) {
  extern __shared__ double learned_cell_sm[];
  d_sweep_cell<3, DIR, IDFX_LEARNED, kHLLD, double>(g, f, ctl, invdt, last_dir, blockIdx.x, learned_cell_sm, lr);
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
    umma::mma_run(taddr, umma::along_columns(umma::smem_addr(As), K), umma::along_columns(umma::smem_addr(Bs), K), 128,
                  N, K);
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
  float* Y = nullptr;  // corrections [3][NOUT][ncell]; null: window by window where the corner EMFs lie
  unsigned long long* counters = nullptr;
  bool ranged = false;
};

namespace idfx {

// the network over every cell of the box, or over a window's
template <bool WINDOW>
static void launch_correct(Engine& e, const LearnedModel& m, const LearnedWindow& win, float* Y, long long room) {
  const LearnedDev L{m.Wp, m.w, m.ranged ? m.fmin : nullptr, m.ranged ? m.fmax : nullptr};
  const LBox box = learned_box(e.g);
  const long long cells = WINDOW ? (long long)win.lines * win.per : box.cells;
  const long long items = (cells + LT - 1) / LT * (WINDOW ? 1 : 3);
  mark_begin(e, kKLearned);
  k_learned_correct<WINDOW><<<(unsigned)(items < e.sms ? items : e.sms), LN, SM_LEARN, e.stream>>>(
      e.g, e.f.Vc32, e.f.Vc, L, e.ctl, box, win, Y, room);
  mark_end(e);
}

// the cell sweep along d over `lines` lines
template <bool WINDOW>
static void launch_sweep_learned(Engine& e, int d, int invdt, int last, long long lines,
                                 const LearnedRecon<WINDOW>& lr) {
  const Geo& g = e.g;
  const int nt = cell_threads(e.sms, [&](int t) { return cell_tiles(g, d, t, 8, lines); });
  const unsigned grid = (unsigned)cell_tiles(g, d, nt, 8, lines);
  const size_t sm = cell_smem_bytes(3, nt, 8);
  mark_begin(e, kKSweepX + d);
  if (d == 0) k_sweep_learned<0, WINDOW><<<grid, nt, sm, e.stream>>>(g, e.f, e.ctl, invdt, last, lr);
  if (d == 1) k_sweep_learned<1, WINDOW><<<grid, nt, sm, e.stream>>>(g, e.f, e.ctl, invdt, last, lr);
  if (d == 2) k_sweep_learned<2, WINDOW><<<grid, nt, sm, e.stream>>>(g, e.f, e.ctl, invdt, last, lr);
  mark_end(e);
}

// the learned sweeps of one stage: the corrections of the three directions,
// then direction after direction (the same InvDt modes as the plain sweeps: 1
// first contribution, 2 accumulate; the last direction folds the CFL
// maximum); states: face states instead.  Without room for the corrections
// of a box, each direction in windows, whose corrections the sweep takes
// before the next window's replace them.
static void launch_learned(Engine& e, int invdt, int fold_max, double* states) {
  const LearnedModel& m = *static_cast<LearnedModel*>(e.learned);
  const Geo& g = e.g;
  if (m.Y) launch_correct<false>(e, m, LearnedWindow{}, m.Y, 0);
  for (int d = 0; d < 3; d++) {
    const int inv = (invdt == 0) ? 0 : (d == 0 ? invdt : 2);
    const int last = fold_max && d == 2;
    const unsigned lines = (unsigned)cell_lines(g, d), per = (unsigned)(g.n[d] + 2);
    if (m.Y) {
      launch_sweep_learned(e, d, inv, last, lines, LearnedRecon<false>{m.Y, 0, LearnedWindow{}, states, m.counters});
      continue;
    }
    float* Y = reinterpret_cast<float*>(e.f.ex);  // ex, ey and ez, one after the other
    const long long room = 6 * g.ncell / NOUT;
    for (unsigned l = 0; l < lines;) {
      const LearnedWindow win = window_from(d, l, lines, per, (unsigned)room);
      launch_correct<true>(e, m, win, Y, room);
      launch_sweep_learned(e, d, inv, last, win.lines, LearnedRecon<true>{Y, room, win, states, m.counters});
      l += win.lines;
    }
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
  cudaFree(m->Y);
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
  int* status = nullptr;       // set by a block whose bounded wait gave up: mapped host memory, read
  int* status_host = nullptr;  // without another copy
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
  launch_chained(h->stream, k_train_tile, n, TT, SM_TRAIN, a);
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
  launch_chained(h->stream, k_train_update, grad ? UPDATE_BLOCKS : 1, 256, 0, grad ? h->part : nullptr, h->cols,
                 h->max_batch, split_batch(B).blocks, h->g, adam, h->ploss, B, loss);
}

int sync_ok(idfx_mlp* h) {
  if (cudaGetLastError() != cudaSuccess) return IDFX_ERR_CUDA;
  if (cudaStreamSynchronize(h->stream) != cudaSuccess) return IDFX_ERR_CUDA;
  if (h->status_host && *(volatile int*)h->status_host) return IDFX_ERR_CUDA;  // a bounded tensor-core wait gave up
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
    ok = ok && cudaFuncSetAttribute(k_learned_correct<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)SM_LEARN) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(k_learned_correct<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)SM_LEARN) == cudaSuccess;
    // no room for the whole box's corrections: window by window (launch_learned)
    if (ok && e.f.Vc32 && cudaMalloc(&m->Y, sizeof(float) * 3 * NOUT * e.g.ncell) != cudaSuccess) {
      m->Y = nullptr;
      cudaGetLastError();
    }
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
            dalloc(h, &h->kmax, NIN);
  ok = ok && cudaHostAlloc(&h->status_host, sizeof(int), cudaHostAllocMapped) == cudaSuccess;
  if (ok) *h->status_host = 0;
  ok = ok && cudaHostGetDevicePointer(reinterpret_cast<void**>(&h->status), h->status_host, 0) == cudaSuccess;
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
  if (h->status_host) cudaFreeHost(h->status_host);
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
