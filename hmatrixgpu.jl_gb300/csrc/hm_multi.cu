// Multi-right-hand-side H-matrix product, plain form (FP32 or FP64 on the CUDA
// cores): Y = H X for up to kRhs right-hand sides per pass.
//
// A pass is W right-hand sides wide (W = 8, 16 or 32, in FP64 4 too: the narrowest
// that holds the pass's columns). XT holds, for every permuted source index and every
// rank row, the W values of that row contiguously (row-major, 4W bytes per row
// in FP32). The matrix is read once per pass and every element feeds W FMAs,
// so the 32-wide form is bound by the CUDA cores' FMA rate (FP64: by the FP64
// pipe at every width) and the 8-wide FP32 one by HBM.
//
// Both passes run the same micro-kernel (slice_product): one warp multiplies
// panels of at most 64 rows with W right-hand sides, a register tile of up to
// 8 x 8 per lane, its operands copied into its own two stages of shared memory,
// so that warps never wait for one another inside a panel. The warps of a CTA
// share a panel by column slices, whose sums meet in shared memory in warp order;
// V items of few columns go to single warps. Results are deterministic.
//
// Measured on a film of 262,144 points (633 M stored entries, FP32), us per product with 32,
// 16 and 8 right-hand sides: 1039, 647 and 558, against 2336 for the form before (CTA-wide
// stages, 4 x 8 or 2 x 16 tiles, panel entries straight from global memory: L1-bound). The
// FMAs alone take 633 at 32 TFMA/s, the entries' bytes 374.
#include <cuda_runtime.h>

#include <type_traits>

#include "hm_device.h"
#include "hm_launch.cuh"
#include "hm_per_device.h"

namespace hm {

constexpr int kRhs = 32;  // right-hand sides per pass at most (row length of XT)
// Warps per CTA of the V pass and of the near/U pass, and CTAs per SM (16 warps of 128
// registers a thread in FP32; FP64 needs more registers for the same tile, and 8 warps keep
// the FP64 pipe busy). More CTAs hide one another's panel starts and ends better, more warps
// read longer runs of each panel row: V pass of a 40,960-point cube, 32 wide, FP32, in us with
// 4 / 8 warps 355 / 400, near/U pass 812 / 663 (film of 262,144: 695 / 719).
constexpr int kVWarps = 4, kDuWarps = 8;
template <typename T, int NW>
constexpr int multi_ctas() {
  return (sizeof(T) == 4 ? 16 : 8) / NW;
}
constexpr int kPanelRows = 64;  // rows of a panel at most

// ticket counters (slots of DevPlan::counter): near/U units, V items of CTAs, of warps
constexpr int kTickets = 3;
__device__ constexpr int kTicket[kTickets] = {0, 1, 8};

// XT rows from X in its own order: X[j + r ldx] goes to XT[sinv[j] W + r]
// (0 for r >= nr). Reads of X are coalesced along j and every XT row is written
// whole; the x-region rows that no source index maps to stay zero (every pass
// width has its own XT, zeroed once). Also re-arms the ticket counters.
template <typename T, int W>
__global__ void permute_multi_kernel(const T *X, int64_t ldx, int nr,
                                     const int32_t *__restrict__ sinv0, int64_t n_src,
                                     T *xt, int32_t *counter) {
  __shared__ T tile[64][W + 1];
  pdl_wait();
  pdl_trigger();
  if (blockIdx.x == 0 && threadIdx.x < kTickets) counter[kTicket[threadIdx.x]] = 0;
  for (int64_t j0 = blockIdx.x * 64ll; j0 < n_src; j0 += gridDim.x * 64ll) {
#pragma unroll
    for (int i = 0; i < W / 4; i++) {  // all of a thread's loads in flight
      const int e = threadIdx.x + i * kThreads, r = e / 64, jj = e % 64;  // consecutive threads: consecutive j
      const int64_t j = j0 + jj;
      tile[jj][r] = (j < n_src && r < nr) ? X[j + r * ldx] : T(0);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 64 * W; e += blockDim.x) {
      const int jj = e / W, r = e % W;
      if (j0 + jj < n_src) xt[static_cast<int64_t>(sinv0[j0 + jj]) * W + r] = tile[jj][r];
    }
    __syncthreads();
  }
}

// 16-byte asynchronous copy global -> shared; zeros when `valid` is false
// (then nothing is read from `src`).
__device__ __forceinline__ void cp16(void *dst, const void *src, bool valid) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <typename T>
struct Elem {
  static constexpr int kVec = 16 / sizeof(T);   // elements of a 16-byte copy
  static constexpr int kStep = 64 / sizeof(T);  // columns per stage: 64 bytes of a panel row
};

// Lane layout of a panel of MT rows x W right-hand sides: NG lanes along the
// right-hand sides (TN each) times RG lanes along the rows (rows rg, rg + RG, ...:
// TR each). FP32: 8 right-hand sides a lane where that leaves 48 or 64 accumulators (16 shared
// loads of 16 bytes per 256 FMAs), 4 otherwise. FP64 is bound by the FP64 pipe, which takes
// as long for an idle lane as for a busy one, and shared loads are cheap beside it: few lanes
// along the rows (4; 8 of a 4-wide pass), so that a panel of any number of rows wastes little.
template <typename T, int W, int MT>
struct LaneTile {
  static constexpr bool F64 = sizeof(T) == 8;
  static constexpr int TN = F64 ? (W >= 8 ? W / 8 : 1) : W == 32 && MT >= 48 ? 8 : 4;
  static constexpr int NG = W / TN, RG = 32 / NG, TR = MT / RG;
  static_assert(TR * RG == MT, "whole rows");
};

// Sets of sums a lane keeps, the four quarters of a stage in turn: narrow FP32 passes have the
// registers, and the shorter chains of additions are closer to the exact sum. By the width alone, so
// that a row's sum does not depend on how its tile's rows are cut.
template <typename T, int W>
constexpr int sum_sets() {
  return sizeof(T) == 8 || W == 32 ? 1 : 32 / W;
}

// Stages of one warp: per stage 64 rows x 64 bytes of the panel, the 16-byte
// pieces of row r swapped by (r / 2) mod 4 (eight consecutive rows then touch all
// banks once), then kStep rows of XT.
template <typename T, int W>
constexpr int stage_bytes() {
  return kPanelRows * 64 + Elem<T>::kStep * W * static_cast<int>(sizeof(T));
}
template <typename T, int W, int NW>
constexpr size_t multi_smem() {
  return static_cast<size_t>(NW) * 2 * stage_bytes<T, W>();
}

__device__ __forceinline__ void lds16(const unsigned char *p, float (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4 *>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void lds16(const unsigned char *p, double (&v)[2]) {
  const double2 a = *reinterpret_cast<const double2 *>(p);
  v[0] = a.x; v[1] = a.y;
}

// A lane's TR x TN sums. In FP32 two neighbouring right-hand sides share a register pair and
// an fma.rn.f32x2, each half rounded as a single FMA is: the FMA rate is the same, but it takes
// half the issue slots (8 x 8 tiles from shared memory: 28 -> 31 TFMA/s), which the copies need.
template <typename T, int TR, int TN>
struct Sums {
  T v[TR][TN];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < TR; i++)
#pragma unroll
      for (int j = 0; j < TN; j++) v[i][j] = T(0);
  }
  struct B {
    T v[TN];
    __device__ __forceinline__ void load(const unsigned char *p) {
      constexpr int VEC = 16 / sizeof(T);
      if constexpr (TN < VEC) {
        v[0] = *reinterpret_cast<const T *>(p);
      } else {
#pragma unroll
        for (int j = 0; j < TN / VEC; j++) {
          T q[VEC];
          lds16(p + j * 16, q);
#pragma unroll
          for (int e = 0; e < VEC; e++) v[j * VEC + e] = q[e];
        }
      }
    }
  };
  __device__ __forceinline__ void add(int i, T a, const B &b) {
#pragma unroll
    for (int j = 0; j < TN; j++) v[i][j] = fma(a, b.v[j], v[i][j]);
  }
  __device__ __forceinline__ void add(const Sums &o) {
#pragma unroll
    for (int i = 0; i < TR; i++)
#pragma unroll
      for (int j = 0; j < TN; j++) v[i][j] += o.v[i][j];
  }
  __device__ __forceinline__ T get(int i, int j) const { return v[i][j]; }
};
template <int TR, int TN>
struct Sums<float, TR, TN> {
  unsigned long long v[TR][TN / 2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < TR; i++)
#pragma unroll
      for (int j = 0; j < TN / 2; j++) v[i][j] = 0ull;
  }
  struct B {
    unsigned long long v[TN / 2];
    __device__ __forceinline__ void load(const unsigned char *p) {
#pragma unroll
      for (int j = 0; j < TN / 4; j++) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(p + j * 16);
        v[2 * j] = q.x;
        v[2 * j + 1] = q.y;
      }
    }
  };
  __device__ __forceinline__ void add(int i, float a, const B &b) {
    unsigned long long aa;
    asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a));
#pragma unroll
    for (int j = 0; j < TN / 2; j++) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[i][j]) : "l"(aa), "l"(b.v[j]));
  }
  __device__ __forceinline__ void add(const Sums &o) {
#pragma unroll
    for (int i = 0; i < TR; i++)
#pragma unroll
      for (int j = 0; j < TN / 2; j++) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v[i][j]) : "l"(o.v[i][j]));
  }
  __device__ __forceinline__ float get(int i, int j) const {
    return __uint_as_float(static_cast<unsigned>(j & 1 ? v[i][j / 2] >> 32 : v[i][j / 2]));
  }
};

// acc = panel x XT over the column stages first, first + step, ... of a panel of m <=
// MT rows (row-major, stride lda, ncols a multiple of 4), by one warp. row_of(c)
// is the XT row of column c, -1 for a zero row; lane l asks for column l of a
// stage, one stage ahead. `buf`: the warp's two stages.
template <typename T, int W, int MT, typename RowOf>
__device__ __forceinline__ void slice_product(const T *A, int64_t lda, int m, int ncols, int first, int step,
                                              const T *xt, unsigned char *buf, RowOf row_of,
                                              Sums<T, LaneTile<T, W, MT>::TR, LaneTile<T, W, MT>::TN> &acc) {
  constexpr int SETS = sum_sets<T, W>();
  Sums<T, LaneTile<T, W, MT>::TR, LaneTile<T, W, MT>::TN> set[SETS];
#pragma unroll
  for (int z = 0; z < SETS; z++) set[z].zero();
  using L = LaneTile<T, W, MT>;
  constexpr int VEC = Elem<T>::kVec, KS = Elem<T>::kStep;
  constexpr int PB = W / VEC;  // 16-byte pieces of an XT row
  constexpr int SB = stage_bytes<T, W>();
  const int lane = threadIdx.x & 31, rg = lane / L::NG, ng = lane - rg * L::NG;
  const int nst = (ncols + KS - 1) / KS;
  const T *arow = A + (lane >> 2) * lda + (lane & 3) * VEC;  // the lane's first row and piece
  int idx = -1;
  auto look_up = [&](int st) {
    const int c = st * KS + lane;
    idx = lane < KS && st < nst ? row_of(c) : -1;
  };
  auto issue = [&](int st, unsigned char *b) {
    const int c0 = st * KS, piece = lane & 3;
    const bool in = c0 + piece * VEC < ncols;
    const T *src = arow + (in ? c0 : 0);
#pragma unroll
    for (int j = 0; j < (MT + 7) / 8; j++) {
      const int r = (lane >> 2) + 8 * j;
      if (r < m) cp16(b + r * 64 + ((piece ^ ((r >> 1) & 3)) << 4), src, in);
      src += 8 * lda;
    }
    unsigned char *xb = b + kPanelRows * 64;
#pragma unroll
    for (int j = 0; j < (KS * PB + 31) / 32; j++) {
      const int e = lane + 32 * j, k = e / PB, p = e - k * PB;
      const int r = __shfl_sync(0xffffffffu, idx, k & 31);
      if (KS * PB % 32 == 0 || e < KS * PB)
        cp16(xb + e * 16, xt + static_cast<int64_t>(r < 0 ? 0 : r) * W + p * VEC, r >= 0);
    }
  };
  if (first < nst) {
    look_up(first);
    issue(first, buf);
    look_up(first + step);
  }
  cp_commit();
  int h = 0;
  for (int st = first; st < nst; st += step, h ^= 1) {
    if (st + step < nst) {
      issue(st + step, buf + (h ^ 1) * SB);
      look_up(st + 2 * step);
    }
    cp_commit();
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();  // every lane's copies of stage st are in place
    const unsigned char *pa = buf + h * SB + rg * 64, *pb = buf + h * SB + kPanelRows * 64 + ng * L::TN * sizeof(T);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      T a[L::TR][VEC];
#pragma unroll
      for (int i = 0; i < L::TR; i++)
        lds16(pa + i * L::RG * 64 + ((q ^ (((rg + i * L::RG) >> 1) & 3)) << 4), a[i]);
#pragma unroll
      for (int k = 0; k < VEC; k++) {
        typename Sums<T, L::TR, L::TN>::B b;
        b.load(pb + (q * VEC + k) * W * sizeof(T));
#pragma unroll
        for (int i = 0; i < L::TR; i++)
          set[q % SETS].add(i, a[i][k], b);
      }
    }
    __syncwarp();  // the stage may be filled again
  }
  cp_wait_all();
  acc = set[0];
#pragma unroll
  for (int z = 1; z < SETS; z++) acc.add(set[z]);
}

// The warps' sums of a panel of m <= MT rows, added in warp order: emit(row, q, sum) for
// every row < m and q < W; consecutive threads get consecutive rows (ROWS) or
// right-hand sides. By the whole CTA, after every warp's product.
template <typename T, int W, int NW, int MT, bool ROWS, typename S, typename Emit>
__device__ __forceinline__ void sum_warps(const S &acc, int m, unsigned char *smem, Emit emit) {
  using L = LaneTile<T, W, MT>;
  constexpr int LD = W + 1;  // row stride of the sums: no bank conflicts either way
  // the sums of all rows at once where they fit the stages, else of half of them
  constexpr int PARTS = static_cast<size_t>(NW) * MT * LD * sizeof(T) <= multi_smem<T, W, NW>() ? 1 : 2;
  constexpr int TRP = (L::TR + PARTS - 1) / PARTS, MP = TRP * L::RG;
  static_assert(static_cast<size_t>(NW) * MP * LD * sizeof(T) <= multi_smem<T, W, NW>(), "sums");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = lane / L::NG, ng = lane - rg * L::NG;
  T *red = reinterpret_cast<T *>(smem);
#pragma unroll
  for (int part = 0; part < PARTS; part++) {
    __syncthreads();  // the stages (or the sums of the part before) are no longer read
#pragma unroll
    for (int i = 0; i < TRP; i++)
      if (part * TRP + i < L::TR)
#pragma unroll
        for (int j = 0; j < L::TN; j++)
          red[(warp * MP + rg + i * L::RG) * LD + ng * L::TN + j] = acc.get(part * TRP + i, j);
    __syncthreads();
    for (int o = tid; o < MP * W; o += NW * 32) {
      const int row = ROWS ? o % MP : o / W, q = ROWS ? o / MP : o % W;
      if (part * MP + row >= m) continue;
      T s = red[row * LD + q];
#pragma unroll
      for (int w = 1; w < NW; w++) s += red[(w * MP + row) * LD + q];
      emit(part * MP + row, q, s);
    }
  }
}

// Row count of the micro-kernel for a panel of m rows: the smallest form that holds them. In
// FP64, where every row counts, there is one for each number of rows per lane (a row test
// inside one 64-row form does not help: the FP64 pipe is as busy with instructions that
// are predicated off); in FP32 four.
template <typename T, int W, int MT = 64, typename F>
__device__ __forceinline__ void with_rows(int m, F f) {
  constexpr int STEP = sizeof(T) == 8 ? LaneTile<T, W, 64>::RG : 16;
  if constexpr (MT > STEP) {
    if (m <= MT - STEP) {
      with_rows<T, W, MT - STEP>(m, f);
      return;
    }
  }
  f(std::integral_constant<int, MT>());
}

// V pass: for every multi-RHS V item
//   out[(I.out + k) * W + r] = sum_j V[k, j] XT[(I.x_off + j) * W + r],
// out = XT (t rows) or the partial rows P of a cut group. Items [0, nbig) by
// CTAs, the others, of few columns, by single warps; first items by number, the
// next from ticket counters.
template <typename T, int W>
__global__ void __launch_bounds__(kVWarps * 32, multi_ctas<T, kVWarps>()) v_multi_kernel(const T *__restrict__ V,
                                                                            const MVItem *__restrict__ items,
                                                                            int32_t nbig, int32_t nitems,
                                                                            T *xt, T *P,
                                                                            int32_t *counter) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  __shared__ int32_t s_ticket;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int32_t ctas = static_cast<int32_t>(gridDim.x);
  unsigned char *buf = dyn_smem + warp * 2 * stage_bytes<T, W>();
  pdl_wait();
  pdl_trigger();
  int32_t u = static_cast<int32_t>(blockIdx.x);
  bool big = u < nbig;
  if (!big) u = nbig + u * kVWarps + warp;
  while (u < nitems) {  // one loop for both kinds, so that the micro-kernels' code is there once
    const MVItem I = items[u];
    T *out = (I.kind == 0 ? xt : P) + static_cast<int64_t>(I.out) * W;
    with_rows<T, W>(I.nrows, [&](auto mt) {
      using L = LaneTile<T, W, mt.value>;
      Sums<T, L::TR, L::TN> acc;
      slice_product<T, W, mt.value>(V + I.v_off, I.stride, I.nrows, I.ncols, big ? warp : 0, big ? kVWarps : 1, xt, buf,
                                    [&](int c) { return c < I.ncols ? I.x_off + c : -1; }, acc);
      if (big) {
        sum_warps<T, W, kVWarps, mt.value, false>(acc, I.nrows, dyn_smem,
                                         [&](int row, int q, T s) { out[static_cast<int64_t>(row) * W + q] = s; });
      } else {
        const int rg = lane / L::NG, ng = lane - rg * L::NG;
#pragma unroll
        for (int i = 0; i < L::TR; i++) {
          const int row = rg + i * L::RG;
          T *o = out + static_cast<int64_t>(row) * W + ng * L::TN;
          if (row < I.nrows)
#pragma unroll
            for (int j = 0; j < L::TN; j++) o[j] = acc.get(i, j);
        }
      }
    });
    if (big) {
      if (tid == 0) s_ticket = next_unit(counter + kTicket[1], ctas, nbig);
      __syncthreads();  // the sums are read, the stages may be filled again
      u = s_ticket;
      if (u >= nbig) {
        big = false;
        u = nbig + static_cast<int32_t>(blockIdx.x) * kVWarps + warp;
      }
    } else {
      int32_t next = 0;
      if (lane == 0) next = nbig + next_unit(counter + kTicket[2], ctas * kVWarps, nitems - nbig);
      u = __shfl_sync(0xffffffffu, next, 0);
    }
  }
}

// t rows of cut groups: pieces summed in order (one warp per row, lane = RHS).
template <typename T, int W>
__global__ void reduce_multi_kernel(const MVReduce *__restrict__ red, int32_t nred, const T *P, T *xt) {
  const int lane = threadIdx.x & 31;
  pdl_wait();
  pdl_trigger();
  if (lane >= W) return;
  for (int32_t e = static_cast<int32_t>(blockIdx.x); e < nred; e += gridDim.x) {
    const MVReduce R = red[e];
    for (int row = threadIdx.x >> 5; row < R.nrows; row += blockDim.x >> 5) {
      T s = T(0);
      const T *p = P + (static_cast<int64_t>(R.p_row) + row) * W + lane;
      const int64_t step = static_cast<int64_t>(R.nrows) * W;
      int j = 0;
      for (; j + 8 <= R.npieces; j += 8) {  // eight loads in flight, added in order
        T v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = p[(j + i) * step];
#pragma unroll
        for (int i = 0; i < 8; i++) s += v[i];
      }
      for (; j < R.npieces; j++) s += p[j * step];
      xt[static_cast<int64_t>(R.t_row + row) * W + lane] = s;
    }
  }
}

// Near/U pass: a run of at most 64 rows of one tile per CTA (first by number, then from a
// ticket counter, tiles with the most columns first).
template <typename T>
struct DuMultiArgs {
  const T *panels;
  const MUnit *units;
  int32_t nunits;
  const int32_t *colmap;  // XT row of every tile column, tile after tile
  const T *xt;
  const int32_t *tmap0;
  T *y;
  int64_t ldy;
  int nr;
  int32_t *counter;
};

// The column map of every tile from its segments: a warp per segment would leave most lanes idle
// on rank columns, so a warp takes a tile and each lane its columns, by binary search.
__global__ void __launch_bounds__(kThreads) colmap_kernel(const TileDesc *__restrict__ tiles, int32_t ntiles,
                                                          const Seg *__restrict__ segs,
                                                          const int64_t *__restrict__ col0,
                                                          int32_t *__restrict__ colmap) {
  const int lane = threadIdx.x & 31;
  for (int64_t t = blockIdx.x * static_cast<int64_t>((kThreads / 32)) + (threadIdx.x >> 5); t < ntiles;
       t += static_cast<int64_t>(gridDim.x) * (kThreads / 32)) {
    const TileDesc d = tiles[t];
    const Seg *S = segs + d.seg0;
    int lo0 = 0;
    for (int c = lane; c < d.ncols; c += 32) {
      int lo = lo0, hi = d.nseg - 1;  // last segment with col0 <= c
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (S[mid].col0 <= c)
          lo = mid;
        else
          hi = mid - 1;
      }
      lo0 = lo;
      colmap[col0[t] + c] = S[lo].vec_off + (c - S[lo].col0);
    }
  }
}

cudaError_t launch_colmap(const TileDesc *tiles, int32_t ntiles, const Seg *segs, const int64_t *col0, int32_t *colmap,
                          cudaStream_t s) {
  colmap_kernel<<<ntiles < 8192 ? (ntiles + (kThreads / 32) - 1) / (kThreads / 32) : 1024, kThreads, 0, s>>>(tiles, ntiles, segs, col0,
                                                                                          colmap);
  return cudaGetLastError();
}

template <typename T, int W>
__global__ void __launch_bounds__(kDuWarps * 32, multi_ctas<T, kDuWarps>()) du_multi_kernel(DuMultiArgs<T> a) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  __shared__ int32_t s_ticket;
  const int tid = threadIdx.x, warp = tid >> 5;
  pdl_wait();
  pdl_trigger();
  for (int32_t u = static_cast<int32_t>(blockIdx.x); u < a.nunits;) {
    const MUnit U = a.units[u];
    const int32_t *map = a.colmap + U.map;
    with_rows<T, W>(U.m, [&](auto mt) {
      using L = LaneTile<T, W, mt.value>;
      Sums<T, L::TR, L::TN> acc;
      slice_product<T, W, mt.value>(a.panels + U.data_off, U.ld, U.m, U.ld, warp, kDuWarps, a.xt,
                                    dyn_smem + warp * 2 * stage_bytes<T, W>(),
                                    [&](int c) { return c < U.ncols ? __ldg(map + c) : -1; }, acc);
      sum_warps<T, W, kDuWarps, mt.value, true>(
          acc, U.m, dyn_smem,
          [&](int row, int q, T s) {
            if (q < a.nr) a.y[a.tmap0[U.row0 + row] + q * a.ldy] = s;
          });
    });
    // (the ticket before was read by all warps before sum_warps' barriers)
    if (tid == 0) s_ticket = next_unit(a.counter + kTicket[0], gridDim.x, a.nunits);
    __syncthreads();  // the sums are read, the stages may be filled again
    u = s_ticket;
  }
}

template <typename T, int W>
static cudaError_t multi_attrs() {
  static PerDevice once;
  return once([] {
    const cudaError_t e = cudaFuncSetAttribute(v_multi_kernel<T, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(multi_smem<T, W, kVWarps>()));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(du_multi_kernel<T, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(multi_smem<T, W, kDuWarps>()));
  });
}

template <typename T, int W>
static cudaError_t run_multi(const DevPlan &p, const T *panels, const T *vdata, T *xt, T *P, const T *X,
                             int64_t ldx, int nr, T *Y, int64_t ldy, int num_sms,
                             cudaStream_t s, cudaEvent_t *ev, int *launches) {
  cudaError_t e = multi_attrs<T, W>();
  if (e != cudaSuccess) return e;
  int gp = static_cast<int>((p.n_src + 63) / 64);
  if (gp > 2048) gp = 2048;
  const bool overlap = may_overlap(sizeof(T) == 8, p.entries, W);
  int nl = 0;
  if (ev) cudaEventRecord(ev[0], s);
  e = launch_pdl(overlap, permute_multi_kernel<T, W>, gp, kThreads, 0, s, X, ldx, nr, p.sinv0, p.n_src, xt, p.counter);
  nl++;
  if (ev) cudaEventRecord(ev[1], s);
  if (e == cudaSuccess && p.nmv > 0) {
    const int32_t nbig = sizeof(T) == 4 ? p.nmv_big : p.nmv;
    e = launch_pdl(overlap, v_multi_kernel<T, W>, num_sms * multi_ctas<T, kVWarps>(), kVWarps * 32,
                   multi_smem<T, W, kVWarps>(), s, vdata, p.mv_items, nbig, p.nmv, xt, P, p.counter);
    nl++;
    if (e == cudaSuccess && p.nmvr > 0) {
      e = launch_pdl(overlap, reduce_multi_kernel<T, W>, p.nmvr < 4096 ? p.nmvr : 4096, kThreads, 0, s, p.mv_reduce, p.nmvr, P,
                     xt);
      nl++;
    }
  }
  if (ev) cudaEventRecord(ev[2], s);
  DuMultiArgs<T> a{panels, p.munits, p.nmunits, p.mcolmap, xt, p.tmap0, Y, ldy, nr, p.counter};
  if (e == cudaSuccess)
    e = launch_pdl(overlap, du_multi_kernel<T, W>, num_sms * multi_ctas<T, kDuWarps>(), kDuWarps * 32,
                   multi_smem<T, W, kDuWarps>(), s, a);
  nl++;
  if (ev) cudaEventRecord(ev[3], s);
  if (launches) *launches = nl;
  return e != cudaSuccess ? e : cudaGetLastError();
}

int rhs_per_pass() { return kRhs; }

int multi_width(bool f64, int nr) { return nr <= 4 && f64 ? 4 : nr <= 8 ? 8 : nr <= 16 ? 16 : kRhs; }

// FP32 passes are as wide as they can be: they read the matrix once. In FP64 a pass's time is
// that of the FP64 pipe, in proportion to its width, beside some 12 us of launches and latency, so the
// columns are split into the widths with the least sum of both. 18 columns in one 32-wide pass / as
// chosen, in us: 2000 points on a circle (0.47 M entries) 104 / one pass, 1000-point cube (0.99 M) 94 / 73
// (16 and 4 wide), film of 30,000 (59 M) 4043 / 2609. The worst seen: circle of 20,000, where V rows are long
// and the pipe is not the bound, 28 columns 911 / 951. A row's sum does not depend on the width.
int multi_pass_columns(bool f64, int64_t left, int64_t entries, int num_sms) {
  if (!f64 || left >= kRhs) return static_cast<int>(left < kRhs ? left : kRhs);
  const double column = static_cast<double>(entries) / (2.0 * num_sms * 1900.0);  // us of the FP64 pipe per column
  double best[kRhs + 1] = {0.0};
  int first[kRhs + 1] = {0};
  for (int r = 1; r <= left; r++) {
    best[r] = 1e300;
    for (int w : {32, 16, 8, 4}) {
      const int n = w < r ? w : r;
      const double t = 12.0 + w * column + best[r - n];
      if (t < best[r]) {
        best[r] = t;
        first[r] = n;
      }
    }
  }
  return first[left];
}

template <typename T>
static cudaError_t run_multi_w(const DevPlan &p, int width, const T *panels, const T *vdata, T *xt, T *P, const T *X,
                               int64_t ldx, int nr, T *Y, int64_t ldy, int num_sms, cudaStream_t s,
                               cudaEvent_t *ev, int *launches) {
  if (nr > width) return cudaErrorInvalidValue;
  switch (width) {
    case 4:
      if constexpr (sizeof(T) == 8)
        return run_multi<T, 4>(p, panels, vdata, xt, P, X, ldx, nr, Y, ldy, num_sms, s, ev, launches);
      return cudaErrorInvalidValue;
    case 8: return run_multi<T, 8>(p, panels, vdata, xt, P, X, ldx, nr, Y, ldy, num_sms, s, ev, launches);
    case 16: return run_multi<T, 16>(p, panels, vdata, xt, P, X, ldx, nr, Y, ldy, num_sms, s, ev, launches);
    case kRhs: return run_multi<T, kRhs>(p, panels, vdata, xt, P, X, ldx, nr, Y, ldy, num_sms, s, ev, launches);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_matvec_multi(bool f64, const DevPlan &p, int width, const void *panels, const void *vdata,
                                void *xt, void *P, const void *X, int64_t ldx, int nr, void *Y,
                                int64_t ldy, int num_sms, cudaStream_t s, cudaEvent_t *ev,
                                int *launches) {
  if (f64)
    return run_multi_w<double>(p, width, static_cast<const double *>(panels), static_cast<const double *>(vdata),
                             static_cast<double *>(xt), static_cast<double *>(P),
                             static_cast<const double *>(X), ldx, nr, static_cast<double *>(Y), ldy,
                             num_sms, s, ev, launches);
  return run_multi_w<float>(p, width, static_cast<const float *>(panels), static_cast<const float *>(vdata),
                          static_cast<float *>(xt), static_cast<float *>(P), static_cast<const float *>(X),
                          ldx, nr, static_cast<float *>(Y), ldy, num_sms, s, ev, launches);
}

}  // namespace hm
