// Flux sweeps with one thread per cell (every direction, 2-D and 3-D): the
// FP64 sweeps, and the FP32 sweeps of the mixed path up to a size.
#pragma once
#include "learned_window.cuh"
#include "mhd_kernels.cuh"

namespace idfx {

// ---------------------------------------------------------------------------
// The lines of cells along the sweep direction (the active cells and one
// ghost cell at each end, for every column of the other two directions
// including the CT extension) are laid end to end, `cols` neighbouring lines
// side by side, and the sequence is cut into tiles of blockDim.x cells that
// overlap by two positions: thread t holds column t % cols of position
// t / cols of its tile.  A thread reconstructs its cell, hands the right-face
// state to the thread of the next position through shared memory, solves the
// face on the left of its cell, hands flux and wave speed to the thread of
// the position before it, and updates its cell - one reconstruction and one
// Riemann problem deep, where the march of one thread along a segment of s
// cells goes through s + 2 and s + 1 of them one after the other.
//   Why: the FP64 pipe bounds these sweeps (seeddiv.cuh), and one warp per
// scheduler already fills it, so what a launch costs is its FP64 work shared
// out evenly.  A march repeats two reconstructions and a face per segment: short
// segments, which fill the GPU at small and middle sizes, repeat half of their
// work and more; long ones leave it idle.  Here the overlap of a tile is the only
// work done twice (2 of 128 positions along x, 2 of 128 / cols across it), at every size.
// PPM needs one position more at the front: the limited value of a face and
// the second difference of a cell are formed once, by the thread of the cell
// on the left, and handed on.
// Measured (both stages of a cycle, x / y / z sweeps): 256^3 PLM + HLLD 27.5 /
// 27.1 / 26.6 -> 25.1 / 25.4 / 25.2 ms against the march, 64^3 0.75 / 0.75 / 0.76
// -> 0.49 / 0.52 / 0.52 ms, 2-D 256^2 0.28 / 0.28 -> 0.14 / 0.15 ms, 2-D 64^2
// 0.10 -> 0.045 ms, 91 x 62 x 45 PPM + HLL (RK3) 3.8 / 3.9 / 3.9 -> 1.5 / 1.7 /
// 1.8 ms (the segments the block chose for itself); with the quotients and roots off the FP64 pipe
// (seeddiv.cuh) 256^3 19.1 / 19.4 / 19.2 ms, at the pipe's rate (81 % busy of
// the 84 % it reaches; 160 registers, 12 warps per multiprocessor; 16 warps at
// 128 registers were 3 % slower), and with less to do for the side of a face
// that is not taken (riemann_hlld) 17.9 / 18.3 / 18.0 ms, 76-80 % busy.  Products emulated on the integer pipe
// beside it (69 issue slots each) took a quarter of the pipe's work away and
// changed the time by -6 to +10 %: the sweeps' instruction stream then waits on itself.
// ---------------------------------------------------------------------------
constexpr int kCellThreads = 128;  // largest block
// blocks per multiprocessor that the registers allow, by the size of the arithmetic type
__host__ __device__ constexpr int cell_resident(size_t size) { return size == 8 ? 3 : 5; }

// whether the FP32 sweep along dir of a launch over `cells` active cells takes
// this form; the others read each value once and win where they fill the GPU.
// Measured, us per sweep, this form against the fastest segment of the march
// (y, z), the tile sweep (large 3-D y, z) or the warp chunks (x):
//   2-D x    64^2 8 / 11, 512^2 15 / 40, 2048^2 149 / 190
//   2-D y    64^2 10 / 10, 512^2 20 / 36 (59 with the segment chosen untimed),
//            1024^2 57 / 58 (78), 2048^2 204 / 159
//   3-D x    32^3 10 / 11, 64^3 20 / 25, 128^3 105 / 113, 192^3 328 / 315
//   3-D y,z  48^3 16, 17 / 15, 22 (17, 33), 64^3 24, 25 / 25, 29 (25, 63), 91 x 62 x 45
//            PPM 40, 42 / 48, 53, 96^3 65, 67 / 42, 53; against the segment
//            chosen untimed 80^3 37, 39 / 34, 67, 96^3 60, 60 / 42, 68, 128^3 132,
//            136 / 96, 117, 160^3 249, 260 / 169, 168 (an untuned z sweep between
//            74^3 and 96^3 would be faster in this form)
// (across x a tile's overlap is 2 of its 16 positions.)  Ensembles the same by
// the cells of all boxes: 20 boxes of 64^2 .. 384^2, 3 cycles 2423 -> 1911 us.
inline bool cell_sweep_wins(int D, int dir, long long cells) {
  if (dir == 0) return D == 2 || cells <= 1ll << 22;
  return cells <= (D == 2 ? 1ll << 20 : 400000ll);
}

// columns side by side: lanes along x are neighbours in memory already.
// Across x, FP64: two share half a 32-byte sector and cost 2 of 64 positions
// (256^3 y and z sweeps within 1 % of the x sweep; four columns the same there
// and 6 % slower at 64^3, eight 4 % slower).  FP32: half the bytes per value
// and less arithmetic to hide them behind; eight columns of 16 positions a
// block of 128 (128^3 y and z sweep 145 us; four columns 172, sixteen of a
// block of 256 142 but 8 % slower at 32^3), fewer in smaller blocks.
__host__ __device__ constexpr int cell_cols(int dir, size_t size, int nt) {
  return dir == 0 ? 1 : size == 8 ? 2 : nt / 16;
}
// block size for a launch of tiles(nt) blocks of nt threads: smaller blocks
// where fewer than two per multiprocessor would leave schedulers without a warp
template <typename Tiles>
inline int cell_threads(int sms, Tiles tiles) {
  int nt = kCellThreads;
  while (nt > 32 && tiles(nt) < 2 * sms) nt /= 2;
  return nt;
}

// lines along dir, and the tiles of nt cells of `lines` of them (all)
__host__ inline long long cell_lines(const Geo& g, int dir) {
  const int a = (dir == 0) ? 1 : 0, b = (dir == 2) ? 1 : 2;
  return (long long)(g.n[a] + 2 * g.ext) * (g.D == 3 ? g.n[b] + 2 * g.ext : 1);
}
__host__ inline long long cell_tiles(const Geo& g, int dir, int nt, size_t size, long long lines) {
  const int cols = cell_cols(dir, size, nt);
  const int lead = (g.order == 4) ? 1 : 0;  // PPM's extra position
  const int step = nt / cols - 2 - lead;
  const long long total = (lines + cols - 1) / cols * (g.n[dir] + 2 + lead);
  return (total - 2 - lead + step - 1) / step;
}
__host__ inline long long cell_tiles(const Geo& g, int dir, int nt, size_t size) {
  return cell_tiles(g, dir, nt, size, cell_lines(g, dir));
}

// shared memory of a block of nt threads: right-face states (PPM: before
// them, face values and second differences), flux x area and wave speed
__host__ __device__ constexpr size_t cell_smem_bytes(int D, int nt, size_t size) {
  return size * (size_t)((2 * D + 1) + (D + 2) + 1) * (size_t)nt;
}

// the learned order (5, 3-D): corrections Y of the PLM states (learned.cu) -
// [3][16][ncell], or those of a window's cells [16][room] -, where the face
// states go instead of the sweep (or null), and the counts of evaluated and
// fallen-back cells
template <bool WINDOW>
struct LearnedRecon {
  static constexpr bool window = WINDOW;
  const float* Y;
  long long room;
  LearnedWindow win;
  double* states;
  unsigned long long* counters;
};

template <int D, int DIR, int ORDER, int SOLVER, typename T, typename LR = LearnedRecon<false>>
__device__ __forceinline__ void d_sweep_cell(const Geo& g, const Fields& f, const Ctl* ctl, int invdt, int last_dir,
                                             unsigned tile, T* sm, const LR& lr = LR{}) {
  if (ctl->done) return;
  using v = Var<D>;
  using dd = Dir<D, DIR>;
  constexpr int NV = v::NV, NU = v::BX1, NS = NV - 1;
  constexpr int H = Recon<ORDER>::H;
  constexpr int E = (ORDER == 4) ? 1 : 0;
  constexpr int A = (DIR == 0) ? 1 : 0, B = (DIR == 2) ? 1 : 2;
  const int nt = (int)blockDim.x, tid = (int)threadIdx.x;
  const int cols = cell_cols(DIR, sizeof(T), nt);
  // (the block's constants become FP32 through from_f64: a conversion
  // instruction would take a turn of the FP64 pipe in every thread, 17 of them and of
  // comparisons per cell where 8 are left)
  T* ss = sm;            // [NS][nt] right-face states
  T* sf = sm + NS * nt;  // [NU + 1][nt] flux x area, wave speed
  const T* W;            // primitives
  if constexpr (sizeof(T) == 8) W = f.Vc;
  else W = f.Vc32;
  const int t = tid / cols, npos = nt / cols;
  // 32-bit indices: a position stands for a cell, of which a device holds
  // fewer than 2^31
  const unsigned nA = (unsigned)(g.n[A] + 2 * g.ext);
  const unsigned nB = (D == 3) ? (unsigned)(g.n[B] + 2 * g.ext) : 1u;
  const unsigned P = (unsigned)(g.n[DIR] + 2 + E);  // positions of a line: cells beg - 1 - E .. end
  const unsigned q = tile * (unsigned)(npos - 2 - E) + (unsigned)t;
  const unsigned bundle = q / P;
  const int p = (int)(q - bundle * P);
  unsigned line = bundle * cols + (unsigned)(tid - t * cols);
  const unsigned lines = LR::window ? lr.win.lines : nA * nB;
  const bool valid = line < lines;
  if constexpr (LR::window) line += lr.win.line0;
  int idx[3];
  idx[DIR] = g.beg[DIR] - 1 - E + p;
  idx[A] = g.beg[A] - g.ext + (int)(valid ? line % nA : 0);
  idx[B] = (D == 3) ? g.beg[B] - g.ext + (int)(valid ? line / nA : 0) : 0;
  const long long cc = cidx(g, idx[2], idx[1], idx[0]);
  const long long sd = g.s[DIR];
  bool active_col = valid && idx[A] >= g.beg[A] && idx[A] < g.end[A];
  if constexpr (D == 3) active_col = active_col && idx[B] >= g.beg[B] && idx[B] < g.end[B];
  const bool update = active_col && t >= 1 + E && t <= npos - 2 && p >= 1 + E && p <= g.n[DIR] + E;
  // what the last phase reads, on its way while the first two compute
  if (update) {
#pragma unroll
    for (int n = 0; n < NU; n++) prefetch_l2(f.Uc + n * g.ncell + cc);
  }
  // ---- reconstruction -------------------------------------------------
  T vl[NV], vr[NV];
#pragma unroll
  for (int n = 0; n < NV; n++) vl[n] = vr[n] = T(0);
  if constexpr (ORDER == 4) {
    T w[NV][5];
    if (valid) {
#pragma unroll
      for (int n = 0; n < NV; n++) {
        if (n == dd::BXn) continue;
        const int s = n < dd::BXn ? n : n - 1;
#pragma unroll
        for (int m = 0; m < 4; m++) w[n][m + 1] = W[n * g.ncell + cc + (m - 1) * sd];
        vr[n] = ppm_face(w[n][1], w[n][2], w[n][3], w[n][4]);
        ss[s * nt + tid] = vr[n];
      }
    }
    __syncthreads();
    if (valid && t >= 1 && p >= 1) {
#pragma unroll
      for (int n = 0; n < NV; n++)
        if (n != dd::BXn) vl[n] = ss[(n < dd::BXn ? n : n - 1) * nt + tid - cols];
    }
    __syncthreads();
    if (valid) {
#pragma unroll
      for (int n = 0; n < NV; n++) {
        if (n == dd::BXn) continue;
        w[n][0] = ppm_diff2(w[n][1], w[n][2], w[n][3]);
        ss[(n < dd::BXn ? n : n - 1) * nt + tid] = w[n][0];
      }
    }
    __syncthreads();
    if (valid && t >= 1 && p >= 1) {
#pragma unroll
      for (int n = 0; n < NV; n++) {
        if (n == dd::BXn) continue;
        const T before = ss[(n < dd::BXn ? n : n - 1) * nt + tid - cols];
        ppm_cell(w[n][1], w[n][2], w[n][3], before, w[n][0], ppm_diff2(w[n][2], w[n][3], w[n][4]), vl[n], vr[n]);
        if (n == v::RHO || n == v::PRS) Recon<4>::ppm_positive(w[n][1], w[n][2], w[n][3], vl[n], vr[n]);
      }
    }
    __syncthreads();
    if (valid) {
#pragma unroll
      for (int n = 0; n < NV; n++)
        if (n != dd::BXn) ss[(n < dd::BXn ? n : n - 1) * nt + tid] = vr[n];
    }
  } else if constexpr (ORDER == 5) {
    bool fall = false;
    if (valid) {
      T cen[NV];
#pragma unroll
      for (int n = 0; n < NV; n++) {
        if (n == dd::BXn && !lr.states) continue;
        const T w0 = f.Vc[n * g.ncell + cc - sd], w1 = f.Vc[n * g.ncell + cc], w2 = f.Vc[n * g.ncell + cc + sd];
        cen[n] = w1;
        Recon<2>::plm(w1, w1 - w0, w2 - w1, false, vl[n], vr[n]);
      }
      const T cs = root(quot(g.gamma * cen[v::PRS], cen[v::RHO])), sb = root(cen[v::RHO]) * cs;
      const float* Y = lr.Y;
      if constexpr (LR::window) Y += window_index(lr.win, line, (unsigned)p);
      else Y += (long long)DIR * 16 * g.ncell + cc;
      const long long out = LR::window ? lr.room : g.ncell;  // from one output to the next
      T cl[NV], cr[NV];
#pragma unroll
      for (int rv = 0; rv < 8; rv++) {
        if (rv == 5) continue;  // normal field: the face value is used
        const int n = rv == 0 || rv == 4 ? rv : (rv < 4 ? 1 : 5) + (DIR + rv - (rv < 4 ? 1 : 5)) % 3;
        const T sc = rv == 0 ? cen[v::RHO] : rv == 4 ? cen[v::PRS] : rv < 4 ? cs : sb;
        cl[n] = vl[n] + f2d_exact(Y[rv * out]) * sc;
        cr[n] = vr[n] + f2d_exact(Y[(8 + rv) * out]) * sc;
      }
      // plain PLM where the stencil is outside the trained range (a NaN) or a
      // corrected density or pressure is not positive
      fall = !(gt0(cl[v::RHO]) && gt0(cl[v::PRS]) && gt0(cr[v::RHO]) && gt0(cr[v::PRS]));
#pragma unroll
      for (int n = 0; n < NV; n++) {
        if (n == dd::BXn) continue;
        if (!fall) {
          vl[n] = cl[n];
          vr[n] = cr[n];
        }
        ss[(n < dd::BXn ? n : n - 1) * nt + tid] = vr[n];
      }
      if (lr.states) {
#pragma unroll
        for (int n = 0; n < NV; n++) {
          lr.states[((long long)DIR * 16 + n) * g.ncell + cc] = vl[n];
          lr.states[((long long)DIR * 16 + 8 + n) * g.ncell + cc] = vr[n];
        }
      }
    }
    // a position belongs to the tile it starts in; the last tile has the rest
    const bool owner = valid && (t < npos - 2 || blockIdx.x == gridDim.x - 1);
    const unsigned fell = __ballot_sync(0xffffffffu, owner && fall);
    if ((tid & 31) == 0 && fell) atomicAdd(lr.counters + 1, (unsigned long long)__popc(fell));
    if (tile == 0 && tid == 0) atomicAdd(lr.counters, (unsigned long long)lines * P);
    if (lr.states) return;
  } else if (valid) {
    const double l3 = g.l3b[DIR];
    const T dxd = from_f64<T>(g.dx[DIR]);
    const bool shk = f.shock && f.shock[cc];
#pragma unroll
    for (int n = 0; n < NV; n++) {
      if (n == dd::BXn) continue;
      T w[2 * H + 1];
#pragma unroll
      for (int m = 0; m <= 2 * H; m++) w[m] = W[n * g.ncell + cc + (m - H) * sd];
      Recon<ORDER>::cell(w, dxd, n == v::RHO || n == v::PRS, vl[n], vr[n], shk, l3);
      ss[(n < dd::BXn ? n : n - 1) * nt + tid] = vr[n];
    }
  }
  __syncthreads();
  // ---- the face on the left of the cell -------------------------------
  const bool face = valid && t >= 1 + E && p >= 1 + E;
  T FA[NU], cm = T(0);
#pragma unroll
  for (int n = 0; n < NU; n++) FA[n] = T(0);
  if (face) {
    T vL[NV];
#pragma unroll
    for (int n = 0; n < NV; n++)
      if (n != dd::BXn) vL[n] = ss[(n < dd::BXn ? n : n - 1) * nt + tid - cols];
    const T bn = from_f64<T>(f.Vs[DIR * g.nface + fidx(g, idx[2], idx[1], idx[0])]);
    vL[dd::BXn] = bn;
    vl[dd::BXn] = bn;
    RiemannOut<D, T> r;
    riemann<D, DIR, SOLVER>(from_f64<T>(g.gamma), vL, vl, r);
    store_emf<D, DIR>(g, f, cc, r, vL, vl);
    if (active_col) {
      const Scale<T> area = scale_by(from_f64<T>(g.A[DIR]));
#pragma unroll
      for (int n = 0; n < NU; n++) {
        FA[n] = scaled(r.F[n], area);
        sf[n * nt + tid] = FA[n];
      }
      cm = r.cmax;
      sf[NU * nt + tid] = cm;
    }
  }
  __syncthreads();
  // ---- flux difference ------------------------------------------------
  double run_max = 0.0;
  if (update) {
    const T dtdV = from_f64<T>(ctl->dtdV);
#pragma unroll
    for (int n = 0; n < NU; n++) {
      const T rhs = -dtdV * (sf[n * nt + tid + cols] - FA[n]);
      f.Uc[n * g.ncell + cc] = f.Uc[n * g.ncell + cc] + to_f64(rhs);
    }
    if (invdt) {
      const double prev = (invdt == 1) ? 0.0 : f.InvDt[cc];
      const T c2 = sf[NU * nt + tid + cols] + cm;
      double inv;
      if constexpr (sizeof(T) == 8) inv = prev + quot(pow2x<-1>(c2), g.dx[DIR]);
      else inv = prev + to_f64(T(0.5) * c2 * (T(1) / from_f64<T>(g.dx[DIR])));
      f.InvDt[cc] = inv;
      if (lt(run_max, inv)) run_max = inv;  // NaN never compares greater
    }
  }
  // CFL maximum: reduced over the warp, then an atomic only where it raises
  // the stored maximum (one atomic per warp on one address would queue)
  if (last_dir && invdt) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, run_max, o);
      if (dbits(w) > dbits(run_max)) run_max = w;  // neither negative nor NaN: ordered as their bits
    }
    unsigned long long* mx = (unsigned long long*)&((Ctl*)ctl)->invdt_max_bits;
    if ((tid & 31) == 0 && (unsigned long long)__double_as_longlong(run_max) > *(volatile unsigned long long*)mx)
      atomic_max_pos(mx, run_max);
  }
}

template <int D, int DIR, int ORDER, int SOLVER, typename T>
__global__ void __launch_bounds__(kCellThreads, cell_resident(sizeof(T)))
    k_sweep_cell(Geo g, Fields f, const Ctl* ctl, int invdt, int last_dir) {
  extern __shared__ double cell_sm[];
  chain_wait();
  d_sweep_cell<D, DIR, ORDER, SOLVER, T>(g, f, ctl, invdt, last_dir, blockIdx.x, reinterpret_cast<T*>(cell_sm));
}

}  // namespace idfx
