// Training step of the correction network: batch assembly, forward, loss and
// backward of 128 samples in one block, on the 5th-generation tensor cores.
#pragma once
#include "learned.cuh"
#include "mhd_kernels.cuh"
#include "umma.cuh"

namespace idfx {
namespace learn {

// BF16 weights as the tensor cores read them, one after the other: W1 (rows
// n = 128, columns k = 224), W2 (128 x 128), W3 (16 x 128), each a canonical
// K-major tile (umma.cuh), so that a block fetches all three with one bulk copy
constexpr int PW1 = 0, PW2 = PW1 + NH * K1, PW3 = PW2 + NH * NH, NPACK = PW3 + NOUT * NH;
static_assert((NPACK * 2) % 16 == 0, "bulk copy size");
// position of parameter p among them, -1 for a bias
__host__ __device__ inline int packed_index(int p) {
  if (p < OB1) return PW1 + (int)umma::kmajor_offset((p - OW1) % NH, (p - OW1) / NH, K1) / 2;
  if (p >= OW2 && p < OB2) return PW2 + (int)umma::kmajor_offset((p - OW2) % NH, (p - OW2) / NH, NH) / 2;
  if (p >= OW3 && p < OB3) return PW3 + (int)umma::kmajor_offset((p - OW3) % NOUT, (p - OW3) / NOUT, NH) / 2;
  return -1;
}

// order-preserving map of floats to unsigned keys (atomic min / max)
__device__ __forceinline__ unsigned fkey(float f) {
  const unsigned b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__host__ __device__ inline float fkey_inv(unsigned k) {
  const unsigned b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  float f;
  memcpy(&f, &b, sizeof(f));
  return f;
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {  // splitmix64 finaliser
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

// x / b, the zero numerators (every velocity feature of the centre cell)
// kept out of the division's slow path: 0 / b as 0 times a quotient
__device__ __forceinline__ float zdiv(float x, float b) {
  const float q = (x == 0.f ? 1.f : x) / b;
  return x == 0.f ? x * q : q;
}

__device__ __forceinline__ float vanleer_f(float dvp, float dvm) {
  return dvp * dvm > 0.f ? 2.f * dvp * dvm / (dvp + dvm) : 0.f;
}

// FP32 snapshots [S][8][nc^3] and face targets [S][3][16][nc^3]
struct Dataset {
  const float *prims, *tgt;
  int S, nc;
  float gamma;
};

// (snapshot, cell, direction) of sample i of a run, from a counter-based
// hash: one sample per lane, since each takes three 64-bit divisions
struct Sample {
  int snap, x, y, z, dir;
};
__device__ __forceinline__ Sample pick(const Dataset& D, unsigned long long seed, long long i) {
  const unsigned nc = (unsigned)D.nc;
  const unsigned long long h = mix64(seed ^ mix64((unsigned long long)i));
  const unsigned long long cell = (h >> 16) % ((unsigned long long)nc * nc * nc);
  const unsigned row = (unsigned)(cell / nc);
  return Sample{(int)(h % (unsigned long long)D.S), (int)(unsigned)(cell - (unsigned long long)row * nc),
                (int)(row % nc), (int)(row / nc), (int)((unsigned)(h >> 48) % 3u)};
}

// Samples first .. first + R - 1 of the warp's picked ones (lane's sample in
// `mine`), by one warp: lane q < 27 holds neighbour q of the 3x3x3 stencil, so
// a variable is one load of nine short rows instead of 27 scattered ones per
// thread, and R samples are in flight at once.
//   feature(r, rv, f)  lane q < 27: feature rv * 27 + q of sample r
//   target(r, t)       lane o < 16: normalised correction target o
template <int R, typename Feature, typename Target>
__device__ __forceinline__ void assemble(const Dataset& D, const Sample& mine, int first, int valid, Feature feature,
                                         Target target) {
  const int lane = threadIdx.x & 31;
  const int nb = lane < 27 ? lane : 13;
  const int o0 = nb % 3 - 1, o1 = nb / 3 % 3 - 1, o2 = nb / 9 - 1;
  const int nc = D.nc;
  const long long ncell = (long long)nc * nc * nc;
  float s[R][8], tg[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    auto of = [&](int x) { return __shfl_sync(0xffffffffu, x, first + r); };
    const int snap = of(mine.snap), d = of(mine.dir);
    int q[3] = {of(mine.x), of(mine.y), of(mine.z)};
    const long long cell = ((long long)q[2] * nc + q[1]) * nc + q[0];
#pragma unroll
    for (int a = 0; a < 3; a++) {  // axis a of the box is axis (a - d) mod 3 of the rotated frame
      const int k = a >= d ? a - d : a - d + 3;
      int x = q[a] + (k == 0 ? o0 : k == 1 ? o1 : o2);
      x += x < 0 ? nc : 0;
      q[a] = x - (x >= nc ? nc : 0);
    }
    const float* P = D.prims + (long long)snap * 8 * ncell + ((long long)q[2] * nc + q[1]) * nc + q[0];
    const bool in = r < valid;
#pragma unroll
    for (int rv = 0; rv < 8; rv++) s[r][rv] = in ? P[rot_var(rv, d) * ncell] : 1.f;
    tg[r] = in && lane < 16 ? D.tgt[(((long long)snap * 3 + d) * 16 + lane) * ncell + cell] : 0.f;
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    float cen[8];
#pragma unroll
    for (int rv = 0; rv < 8; rv++) cen[rv] = __shfl_sync(0xffffffffu, s[r][rv], 13);
    const float cs = sqrtf(D.gamma * cen[4] / cen[0]), sb = sqrtf(cen[0]) * cs;
    const float sc[8] = {cen[0], cs, cs, cs, cen[4], sb, sb, sb};
    float w0 = 0.f, w1 = 0.f, w2 = 0.f, scale = 1.f;  // of lane's target variable
#pragma unroll
    for (int rv = 0; rv < 8; rv++) {
      const float v = s[r][rv];
      float f;
      if (rv == 0 || rv == 4) f = v / cen[rv] - 1.f;
      else if (rv < 4) f = zdiv(v - cen[rv], cs);
      else f = zdiv(v, sb);
      feature(r, rv, f);
      const float b = __shfl_sync(0xffffffffu, v, 12), a = __shfl_sync(0xffffffffu, v, 14);
      if ((lane & 7) == rv) {
        w0 = b;
        w1 = cen[rv];
        w2 = a;
        scale = sc[rv];
      }
    }
    const float dd = vanleer_f(w2 - w1, w1 - w0);
    target(r, (tg[r] - (lane < 8 ? w1 - 0.5f * dd : w1 + 0.5f * dd)) / scale);
  }
}

// ---------------------------------------------------------------------------
// One block of 512 threads, 128 samples at a time; other blocks of the launch
// assemble the next step's samples meanwhile (they need nothing of this step),
// so that the gather - as long as the rest together - costs no time of its
// own.  What bounds a training step is not its arithmetic (2.3 GFLOP at batch
// 8192) but the passes: as separate GEMMs, activations, loss and column sums
// it was sixteen launches that moved every activation through memory several
// times, plus 3.5 million atomics on 432 addresses for the feature range.
// Here the samples never leave the chip:
// features, activations and their gradients are BF16 tiles in shared memory,
// pre-activations and products FP32 in tensor memory, and a tile read along
// its columns (K-major) in the forward pass is read along its rows (MN-major)
// where its transpose is needed.  Per block:
//   features -> Z1 -> H1 -> Z2 -> H2 -> Y -> loss, dY
//   dZ2 = (dY W3^T) silu'(Z2);  dZ1 = (dZ2 W2^T) silu'(Z1)
//   dW3 = H2^T dY, dW2 = H1^T dZ2, dW1 = X^T dZ1
// The block's gradients go to its own slot, its dY and dZ in FP32 to columns
// whose sums are the biases' gradients; k_train_update sums both.  How a
// batch is shared out (Split) and in which order everything is summed depends
// on the batch size alone, not on timing or on the device: Adam turns the
// last bits of a gradient near zero into steps of full size, so a training
// run is only as repeatable as its sums.
// Measured, with the copies around them: sixteen steps at batch 8192 8351 ->
// 876 us, 833 with the status word in mapped memory, 786 with each launch in
// place while the one before ends; at 256 7252 -> 719 -> 613 us; loss and
// gradients of a given batch of 8192 437 -> 69 us.  With the gather inside the
// computing blocks this launch took 105 us (256 threads) or 78 us (512), beside
// them 30 us.
// ---------------------------------------------------------------------------
constexpr int TR = 128;  // samples of a block
constexpr int TT = 512;  // its threads: four warps per 32 samples, a quarter of the columns each
constexpr int TQ = TT / 128;
constexpr size_t TS_X = 0;                                   // features 128 x 224
constexpr size_t TS_W = TS_X + (size_t)TR * K1 * 2;          // packed weights; W1's place then holds H2
constexpr size_t TS_H2 = TS_W;
constexpr size_t TS_W2 = TS_W + (size_t)PW2 * 2, TS_W3 = TS_W + (size_t)PW3 * 2;
constexpr size_t TS_H1 = TS_W + (size_t)NPACK * 2;           // layer-1 output 128 x 128
constexpr size_t TS_D = TS_H1 + (size_t)TR * NH * 2;         // dZ2, then dZ1
constexpr size_t TS_DY = TS_D + (size_t)TR * NH * 2;         // dY 128 x 16
constexpr size_t TS_B = TS_DY + (size_t)TR * NOUT * 2;       // biases
constexpr size_t TS_M = TS_B + (size_t)(2 * NH + NOUT) * 4;  // mbarriers, TMEM slot, losses
constexpr size_t SM_TRAIN = TS_M + 32 + 2 * 8 * (TT / 32);
static_assert(TS_H2 + (size_t)TR * NH * 2 <= TS_W2, "H2 in W1's place");
static_assert(NOUT / TQ == 4, "outputs of a thread");
static_assert(TS_W % 128 == 0 && TS_W2 % 128 == 0 && TS_W3 % 128 == 0 && TS_H1 % 128 == 0 && TS_D % 128 == 0 &&
                  TS_DY % 128 == 0,
              "operand alignment");
static_assert(SM_TRAIN <= 227 * 1024, "training tile does not fit in shared memory");
// tensor memory columns
constexpr uint32_t TC_Z1 = 0, TC_Z2 = 128, TC_P = 256, TC_W2 = 384, TC_W1 = 0, TC_W3 = 224;

// an assembled tile in global memory: the feature tile as the tensor cores
// read it, then the targets
struct Tile {
  __nv_bfloat16 X[TR * K1];
  float T[TR * NOUT];
};
static_assert(sizeof(Tile) % 128 == 0 && TR * K1 * 2 % 16 == 0, "bulk copies of tiles");

// A batch of B samples over blocks: chunks of 64 samples, in up to 64 blocks
// of `chunks` chunks each (two from 256 samples to 8192 in whole pairs of
// chunks, else more; one block below four chunks); a block takes its samples
// in tiles of up to 128.
struct Split {
  int chunks, blocks, tiles;  // chunks and tiles of a block
  __host__ __device__ int first(int block, int tile) const { return block * chunks * 64 + tile * TR; }
  __host__ __device__ int rows(int block, int tile, int B) const {
    const int end = (block + 1) * chunks * 64, n = (end < B ? end : B) - first(block, tile);
    return n < 0 ? 0 : n < TR ? n : TR;
  }
};
__host__ inline Split split_batch(int B) {
  const int n = (B + 63) / 64;
  Split s;
  s.chunks = n;
  if (n >= 4) {
    const int most = n / 2 < 64 ? n / 2 : 64;
    s.chunks = (n + most - 1) / most;
  }
  s.blocks = (n + s.chunks - 1) / s.chunks;
  s.tiles = (s.chunks + 1) / 2;
  return s;
}
constexpr int MAX_BLOCKS = 64;

struct TrainArgs {
  int compute;              // blocks that compute; the blocks after them assemble
  int B;
  Split split;
  const __nv_bfloat16* Wp;  // packed weights
  const float* w;           // FP32 parameters (biases)
  const Tile* tiles;        // assembled batch, or null: X, T
  const __nv_bfloat16* X;   // features [B][K1] and targets [B][NOUT] (T null: outputs only)
  const float* T;
  Tile* next;               // assembled by the blocks after the computing ones
  Dataset D;
  unsigned long long seed;
  long long base;
  float* Y;          // outputs [B][NOUT] (forward only), or null
  float* part;       // weight gradients of every block [blocks][NPARAM], or null: no backward pass
  float* cols;       // dZ1, dZ2, dY of every sample: columns [NH + NH + NOUT][ld]
  int ld;
  double* loss;      // per block: summed squared error, summed squared targets; or null
  unsigned *kmin, *kmax;  // feature range, or null
  int* status;       // set when a bounded wait gave up (the host's memory, mapped)
};

// eight BF16 values of row r, columns c .. c + 7 of a tile with C columns
__device__ __forceinline__ void put8(unsigned char* tile, int r, int c, int C, const float* v) {
  alignas(16) __nv_bfloat162 t[4];
#pragma unroll
  for (int i = 0; i < 4; i++) t[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(tile + umma::kmajor_offset(r, c, C)) = *reinterpret_cast<const uint4*>(t);
}

// 128 samples of a batch into a tile, and the range of their features
__device__ __forceinline__ void assemble_tile(const TrainArgs& a, int block, unsigned char* sm) {
  unsigned char* Xs = sm;
  float* Ts = reinterpret_cast<float*>(sm + sizeof(__nv_bfloat16) * TR * K1);
  unsigned* rng = reinterpret_cast<unsigned*>(sm + sizeof(Tile));  // min keys, max keys
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int i0 = a.split.first(block / a.split.tiles, block % a.split.tiles);
  const int rows = a.split.rows(block / a.split.tiles, block % a.split.tiles, a.B);
  for (int e = tid; e < NIN; e += TT) {
    rng[e] = 0xffffffffu;
    rng[NIN + e] = 0u;
  }
  __syncthreads();
  constexpr int R = 4;
  unsigned lo[8], hi[8];
#pragma unroll
  for (int rv = 0; rv < 8; rv++) {
    lo[rv] = 0xffffffffu;
    hi[rv] = 0u;
  }
  const int w0 = warp * (TR / (TT / 32));  // this warp's 16 samples
  const Sample mine = pick(a.D, a.seed, a.base + i0 + w0 + (lane & (TR / (TT / 32) - 1)));
  for (int r0 = w0; r0 < w0 + TR / (TT / 32); r0 += R) {
    const int valid = min(R, rows - r0);
    assemble<R>(
        a.D, mine, r0 - w0, valid,
        [&](int r, int rv, float f) {
          const bool in = r < valid;
          if (lane < 27)
            *reinterpret_cast<__nv_bfloat16*>(Xs + umma::kmajor_offset(r0 + r, rv * 27 + lane, K1)) =
                __float2bfloat16(in ? f : 0.f);
          if (in) {
            lo[rv] = min(lo[rv], fkey(f));
            hi[rv] = max(hi[rv], fkey(f));
          }
        },
        [&](int r, float t) {
          if (lane < 16) Ts[(r0 + r) * NOUT + lane] = r < valid ? t : 0.f;
          if (lane == 16) *reinterpret_cast<uint4*>(Xs + umma::kmajor_offset(r0 + r, NIN, K1)) = make_uint4(0u, 0u, 0u, 0u);
        });
  }
  if (a.kmin && lane < 27) {
#pragma unroll
    for (int rv = 0; rv < 8; rv++) {
      atomicMin(rng + rv * 27 + lane, lo[rv]);
      atomicMax(rng + NIN + rv * 27 + lane, hi[rv]);
    }
  }
  __syncthreads();
  uint4* out = reinterpret_cast<uint4*>(a.next + block);
  for (int e = tid; e < (int)(sizeof(Tile) / 16); e += TT) out[e] = reinterpret_cast<const uint4*>(sm)[e];
  if (a.kmin)
    for (int e = tid; e < NIN; e += TT) {
      atomicMin(a.kmin + e, rng[e]);
      atomicMax(a.kmax + e, rng[NIN + e]);
    }
}

__device__ __forceinline__ void train_tile(const TrainArgs& a, unsigned char* sm) {
  unsigned char *Xs = sm + TS_X, *H1 = sm + TS_H1, *H2 = sm + TS_H2, *Ds = sm + TS_D, *DY = sm + TS_DY;
  float* bs = reinterpret_cast<float*>(sm + TS_B);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + TS_M);  // tensor core, copies
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + TS_M + 16);
  double* wl = reinterpret_cast<double*>(sm + TS_M + 32);  // losses of the warps
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = 32 * (warp & 3) + lane, quarter = warp >> 2;
  const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
  const int block = blockIdx.x;
  if (warp == 0) umma::tmem_alloc(slot, 512);
  // the first tile's copies: all weights, its features where they are assembled;
  // of a later tile W1 again (H2 took its place)
  auto fetch = [&](int t) {
    const uint32_t wbytes = (t == 0 ? NPACK : PW2) * 2;
    mbar_expect(bar + 1, wbytes + (a.tiles ? TR * K1 * 2 : 0));
    bulk_to_smem(sm + TS_W, a.Wp, wbytes, bar + 1);
    if (a.tiles) bulk_to_smem(Xs, a.tiles[block * a.split.tiles + t].X, TR * K1 * 2, bar + 1);
  };
  if (tid == 0) {
    umma::mbar_init1(bar);
    mbar_init(bar + 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fetch(0);
  }
  for (int e = tid; e < NH; e += TT) {
    bs[e] = a.w[OB1 + e];
    bs[NH + e] = a.w[OB2 + e];
  }
  if (tid < NOUT) bs[2 * NH + tid] = a.w[OB3 + tid];
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *slot;
  uint32_t phase = 0;
  // the tiles written so far to the tensor core, `issue` by one thread, every
  // thread waits (bounded) for it
  auto tensor = [&](auto issue) -> bool {
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (tid == 0) {
      issue();
      umma::mma_commit(bar);
    }
    const bool w = umma::mbar_wait_bounded(bar, phase, umma::kMmaSpin);
    phase ^= 1u;
    const bool ok = __syncthreads_and(w) != 0;
    umma::fence_after_sync();
    return ok;
  };
  // SiLU(acc + bias) -> BF16 operand of the next layer, this thread's quarter of the columns
  auto hidden = [&](uint32_t d_col, const float* bias, unsigned char* out) {
    for (int c = NH / TQ * quarter; c < NH / TQ * (quarter + 1); c += 16) {
      float x[16];
      umma::tmem_ld16(tmem + lanes + d_col + (uint32_t)c, x);
#pragma unroll
      for (int i = 0; i < 16; i++) x[i] = silu_f(x[i] + bias[c + i]);
      put8(out, row, c, NH, x);
      put8(out, row, c + 8, NH, x + 8);
    }
  };
  const uint32_t xa = umma::smem_addr(Xs), w1 = umma::smem_addr(sm + TS_W), w2 = umma::smem_addr(sm + TS_W2),
                 w3 = umma::smem_addr(sm + TS_W3), h1 = umma::smem_addr(H1), h2 = umma::smem_addr(H2),
                 ds = umma::smem_addr(Ds), dy = umma::smem_addr(DY);
  using umma::along_columns;
  using umma::along_rows;
  float* part = a.part ? a.part + (long long)block * NPARAM : nullptr;
  double l = 0.0, l0 = 0.0;
  bool ok = true;
  int t = 0;
  for (; t < a.split.tiles && ok; t++) {
    const int i0 = a.split.first(block, t), rows = a.split.rows(block, t, a.B);
    if (t > 0 && rows == 0) break;
    if (t > 0 && tid == 0) {  // every MMA and every thread's reads of the last tile are done (see the end of the loop)
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      fetch(t);
    }
    if (!a.tiles) {  // features of a given batch
      const bool aligned = (reinterpret_cast<uintptr_t>(a.X) & 15) == 0;  // rows are 448 bytes
      // eight rows of a 16-byte column group: one core matrix, a contiguous 128 bytes
      for (int e = tid; e < TR * (K1 / 8); e += TT) {
        const int r = (e & 7) + 8 * (e / (8 * (K1 / 8))), c = 8 * (e / 8 % (K1 / 8));
        const __nv_bfloat16* src = a.X + (long long)(i0 + r) * K1 + c;
        alignas(16) __nv_bfloat16 v[8];
        if (r < rows && aligned) {
          *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(src);
        } else {
#pragma unroll
          for (int i = 0; i < 8; i++) v[i] = r < rows ? src[i] : __float2bfloat16(0.f);
        }
        *reinterpret_cast<uint4*>(Xs + umma::kmajor_offset(r, c, K1)) = *reinterpret_cast<const uint4*>(v);
      }
    }
    // dZ = acc silu'(Z) -> BF16 tile, and in FP32 to its column (from `first`)
    auto backward = [&](uint32_t z_col, const float* bias, int first) {
      for (int c = NH / TQ * quarter; c < NH / TQ * (quarter + 1); c += 16) {
        float x[16], z[16];
        umma::tmem_ld16(tmem + lanes + TC_P + (uint32_t)c, x);
        umma::tmem_ld16(tmem + lanes + z_col + (uint32_t)c, z);
#pragma unroll
        for (int i = 0; i < 16; i++) x[i] *= dsilu_f(z[i] + bias[c + i]);
        put8(Ds, row, c, NH, x);
        put8(Ds, row, c + 8, NH, x + 8);
        if (row < rows) {
#pragma unroll
          for (int i = 0; i < 16; i++) a.cols[(long long)(first + c + i) * a.ld + i0 + row] = x[i];
        }
      }
    };
    // the block's weight gradients so far, where the next products add to them
    auto resume = [&](uint32_t d_col, int c, const float* from, int stride, int n) {
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; i++) x[i] = c + i < n ? from[(c + i) * stride] : 0.f;
      umma::tmem_st16(tmem + lanes + d_col + (uint32_t)c, x);
    };
    ok = __syncthreads_and(mbar_wait(bar + 1, (uint32_t)(t & 1))) != 0;
    // ---- forward ------------------------------------------------------
    ok = ok && tensor([&] { umma::mma_run(tmem + TC_Z1, along_columns(xa, K1), along_columns(w1, K1), TR, NH, K1); });
    if (ok) {
      hidden(TC_Z1, bs, H1);
      ok = tensor([&] { umma::mma_run(tmem + TC_Z2, along_columns(h1, NH), along_columns(w2, NH), TR, NH, NH); });
    }
    if (ok) {
      hidden(TC_Z2, bs + NH, H2);
      ok = tensor([&] { umma::mma_run(tmem + TC_P, along_columns(h2, NH), along_columns(w3, NH), TR, NOUT, NH); });
    }
    // ---- loss, dY: a quarter of the outputs per thread -------------------
    if (ok) {
      constexpr int NQ = NOUT / TQ;
      float all[16], y[NQ];
      umma::tmem_ld16(tmem + lanes + TC_P, all);
#pragma unroll
      for (int i = 0; i < NQ; i++) {
        const int o = NQ * quarter + i;
#pragma unroll
        for (int k = 0; k < TQ; k++)
          if (quarter == k) y[i] = all[NQ * k + i];
        y[i] += bs[2 * NH + o];
        if (a.Y && row < rows) a.Y[(long long)(i0 + row) * NOUT + o] = y[i];
        const bool in = row < rows && !loss_masked(o);
        float tg = 0.f;
        if (in && a.loss)
          tg = a.tiles ? a.tiles[block * a.split.tiles + t].T[row * NOUT + o] : a.T[(long long)(i0 + row) * NOUT + o];
        const float r = in ? y[i] - tg : 0.f;
        const double rd = f2d_exact(r), td = f2d_exact(tg);
        l += rd * rd;
        if (!part) l0 += td * td;
        y[i] = zdiv(2.f * r, (float)a.B);
        if (part && row < rows) a.cols[(long long)(2 * NH + o) * a.ld + i0 + row] = y[i];
      }
      if (part) {
        alignas(8) __nv_bfloat162 d[2] = {__floats2bfloat162_rn(y[0], y[1]), __floats2bfloat162_rn(y[2], y[3])};
        *reinterpret_cast<uint2*>(DY + umma::kmajor_offset(row, NQ * quarter, NOUT)) =
            *reinterpret_cast<const uint2*>(d);
      }
    }
    if (!part) {
      __syncthreads();
      continue;
    }
    // ---- backward -------------------------------------------------------
    // dZ2's product: dY . W3 (rows n = out of the packed W3, read along them)
    ok = ok && tensor([&] { umma::mma_run(tmem + TC_P, along_columns(dy, NOUT), along_rows(w3, NH), TR, NH, NOUT); });
    if (ok) {
      backward(TC_Z2, bs + NH, NH);
      if (t > 0) {
        __syncthreads();  // Z2 is read; dW3 takes columns of it
        for (int k = NH / TQ * quarter; k < NH / TQ * (quarter + 1); k += 16)
          resume(TC_W2, k, part + OW2 + row, NH, NH);
        if (quarter == 0) resume(TC_W3, 0, part + OW3 + row * NOUT, 1, NOUT);
      }
      // dZ1's product dZ2 . W2, and with it dW3 (rows: hidden, into Z2's place) and dW2 (rows: out)
      ok = tensor([&] {
        umma::mma_run(tmem + TC_P, along_columns(ds, NH), along_rows(w2, NH), TR, NH, NH);
        umma::mma_run(tmem + TC_W3, along_rows(h2, NH), along_rows(dy, NOUT), NH, NOUT, TR, t > 0);
        umma::mma_run(tmem + TC_W2, along_rows(ds, NH), along_rows(h1, NH), NH, NH, TR, t > 0);
      });
    }
    if (ok) {
      backward(TC_Z1, bs, 0);
      if (t > 0) {
        __syncthreads();  // Z1 is read; dW1 takes its place
        for (int k = 16 * quarter; k < K1; k += 16 * TQ) resume(TC_W1, k, part + OW1 + row, NH, NIN);
      }
      ok = tensor([&] { umma::mma_run(tmem + TC_W1, along_rows(ds, NH), along_rows(xa, K1), NH, K1, TR, t > 0); });
    }
    if (ok) {  // lane = a hidden unit: dW1 [k][n], dW2 [in][out], dW3 [hidden][out]
      for (int k = 16 * quarter; k < K1; k += 16 * TQ) {
        float x[16];
        umma::tmem_ld16(tmem + lanes + TC_W1 + (uint32_t)k, x);
#pragma unroll
        for (int i = 0; i < 16; i++)
          if (k + i < NIN) part[OW1 + (k + i) * NH + row] = x[i];
      }
      for (int k = NH / TQ * quarter; k < NH / TQ * (quarter + 1); k += 16) {
        float x[16];
        umma::tmem_ld16(tmem + lanes + TC_W2 + (uint32_t)k, x);
#pragma unroll
        for (int i = 0; i < 16; i++) part[OW2 + (k + i) * NH + row] = x[i];
      }
      if (quarter == 0) {
        float x[16];
        umma::tmem_ld16(tmem + lanes + TC_W3, x);
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          *reinterpret_cast<float4*>(part + OW3 + row * NOUT + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
      }
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
  }
  if (a.loss) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      l += __shfl_down_sync(0xffffffffu, l, o);
      if (!part) l0 += __shfl_down_sync(0xffffffffu, l0, o);
    }
    if (lane == 0) {
      wl[warp] = l;
      wl[TT / 32 + warp] = l0;
    }
    __syncthreads();
    if (tid < 2) {
      double s = 0.0;
      for (int q = 0; q < TT / 32; q++) s += wl[TT / 32 * tid + q];
      a.loss[2 * block + tid] = s;
    }
  }
  if (!ok && tid == 0) {
    *(volatile int*)a.status = 1;
    __threadfence_system();
    mbar_wait(bar + 1, (uint32_t)((t - 1) & 1));  // no copy may land after the block has gone
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

__global__ void __launch_bounds__(TT, 1) k_train_tile(TrainArgs a) {
  extern __shared__ __align__(128) unsigned char train_sm[];
  chain_wait();
  if ((int)blockIdx.x < a.compute) train_tile(a, train_sm);
  else assemble_tile(a, (int)blockIdx.x - a.compute, train_sm);
}
static_assert(NPARAM % 4 == 0 && OW3 % 4 == 0, "float4 stores of dW3");
static_assert(K1 % 16 == 0 && NH / TQ % 16 == 0, "columns in whole groups");

// Adam's factors of one step
struct AdamArgs {
  float lr, b1, b2, eps, bc1, bc2;
  float *w, *m, *v;
  __nv_bfloat16* Wp;
};

__device__ __forceinline__ void adam_step(const AdamArgs& adam, int p, float gp) {
  if (!adam.w) return;
  const float mp = adam.b1 * adam.m[p] + (1.f - adam.b1) * gp;
  const float vp = adam.b2 * adam.v[p] + (1.f - adam.b2) * gp * gp;
  adam.m[p] = mp;
  adam.v[p] = vp;
  const float wp = adam.w[p] - adam.lr * (mp / adam.bc1) / (sqrtf(vp / adam.bc2) + adam.eps);
  adam.w[p] = wp;
  const int at = packed_index(p);
  if (at >= 0) adam.Wp[at] = __float2bfloat16(wp);
}

// blocks of k_train_update: one per bias, then 64 weights each
constexpr int NBIAS = 2 * NH + NOUT;
constexpr int UPDATE_BLOCKS = NBIAS + OB1 / 64 + NH * NH / 64 + NH * NOUT / 64;
static_assert(OB1 % 64 == 0 && OW2 % 64 == 0 && OB2 % 64 == 0 && OW3 % 64 == 0 && OB3 % 64 == 0, "whole groups of 64");

// Gradients of the batch and, where adam.w is set, the Adam step with the BF16
// weights refreshed; block 0 also sums the losses (/ B).
//   weights  the blocks' gradients added one after the other in block order:
//            four threads per parameter bring them in (12 MB a step at batch 8192, from L2),
//            one adds them up
//   biases   the column sum of dZ or dY: thread t every 256th sample from t on,
//            then a tree over the threads
//   (no __restrict__: the launch before writes part, cols and loss while this
//   one's blocks are resident, see launch_chained)
__global__ void __launch_bounds__(256) k_train_update(const float* part, const float* cols, int ld, int blocks,
                                                      float* g, AdamArgs adam, const double* loss, int B,
                                                      double* loss_out) {
  __shared__ float in[MAX_BLOCKS][64];
  chain_wait();
  const int tid = threadIdx.x;
  if (part && blockIdx.x < NBIAS) {
    const int n = blockIdx.x;
    const float* x = cols + (long long)n * ld;
    float* red = &in[0][0];
    float s = 0.f;
    int m = tid;
    for (; m + 7 * 256 < B; m += 8 * 256) {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = x[m + 256 * k];
#pragma unroll
      for (int k = 0; k < 8; k++) s += v[k];
    }
    for (; m < B; m += 256) s += x[m];
    red[tid] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
      if (tid < w) red[tid] += red[tid + w];
      __syncthreads();
    }
    if (tid == 0) {
      const int p = n < NH ? OB1 + n : n < 2 * NH ? OB2 + n - NH : OB3 + n - 2 * NH;
      g[p] = red[0];
      adam_step(adam, p, red[0]);
    }
  } else if (part) {
    int p0 = ((int)blockIdx.x - NBIAS) * 64;  // among the weights
    if (p0 >= OB1) p0 += OW2 - OB1;
    if (p0 >= OB2) p0 += OW3 - OB2;
    const int q = tid >> 6, i = tid & 63, p = p0 + i;
    float x[MAX_BLOCKS / 4];
#pragma unroll
    for (int k = 0; k < MAX_BLOCKS / 4; k++) {
      const int t = MAX_BLOCKS / 4 * q + k;
      x[k] = t < blocks ? part[(long long)t * NPARAM + p] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < MAX_BLOCKS / 4; k++) in[MAX_BLOCKS / 4 * q + k][i] = x[k];
    __syncthreads();
    if (q == 0) {
      float gp = 0.f;
      for (int t = 0; t < blocks; t++) gp += in[t][i];
      g[p] = gp;
      adam_step(adam, p, gp);
    }
  }
  if (blockIdx.x == 0 && loss && tid < 64) {  // warp 0 the loss, warp 1 the squared targets
    const int k = tid >> 5;
    double s = 0.0;
    for (int t = tid & 31; t < blocks; t += 32) s += loss[2 * t + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((tid & 31) == 0) loss_out[k] = s / B;
  }
}

// the BF16 weights of FP32 parameters, packed (the pad columns of W1 zero)
__global__ void k_pack_weights(const float* __restrict__ w, __nv_bfloat16* __restrict__ Wp) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < NPARAM) {
    const int at = packed_index(p);
    if (at >= 0) Wp[at] = __float2bfloat16(w[p]);
  }
  if (p < NH * (K1 - NIN)) Wp[PW1 + umma::kmajor_offset(p % NH, NIN + p / NH, K1) / 2] = __float2bfloat16(0.f);
}

// a batch in global memory: X [B][K1], T [B][NOUT]
__global__ void __launch_bounds__(256) k_make_batch(Dataset D, unsigned long long seed, long long base, int B,
                                                    __nv_bfloat16* __restrict__ X, float* __restrict__ T) {
  constexpr int R = 4;
  const int lane = threadIdx.x & 31;
  const int r0 = ((int)blockIdx.x * 8 + (int)(threadIdx.x >> 5)) * R;
  const int valid = min(R, B - r0);
  if (valid <= 0) return;
  const Sample mine = pick(D, seed, base + r0 + (lane & (R - 1)));
  assemble<R>(
      D, mine, 0, valid,
      [&](int r, int rv, float f) {
        if (r < valid && lane < 27) X[(long long)(r0 + r) * K1 + rv * 27 + lane] = __float2bfloat16(f);
      },
      [&](int r, float t) {
        if (r >= valid) return;
        if (lane < 16) T[(long long)(r0 + r) * NOUT + lane] = t;
        if (lane < K1 - NIN) X[(long long)(r0 + r) * K1 + NIN + lane] = __float2bfloat16(0.f);
      });
}

}  // namespace learn
}  // namespace idfx
