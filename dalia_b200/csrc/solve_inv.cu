// Triangular sweeps with precomputed inverses of the diagonal factor blocks.
//
// With V_i = L_ii^-1 available, a sweep over n blocks is n dependent steps of
// two dense matrix-vector products each,
//   forward   y_i = V_i (b_i - L_{i,i-1} y_{i-1}),
//   backward  x_i = V_i^T (y_i - L_{i+1,i}^T x_{i+1} - Ab_i^T x_a),
// instead of ceil(b/64) dependent tile solves per block.  One persistent
// cooperative launch covers a range of steps of every instance of a batch:
// the CTAs share the rows (forward) or 16-column strips (backward) of a
// product evenly and meet at a grid barrier between the two products of a
// step.
//
// A step's bytes take 4 us at full bandwidth for b = 1500, so latency counts:
// one CTA of 16 warps per SM (a barrier of 148 arrivals), the vector staged
// in shared memory once per product, every result finished inside one CTA (a
// row by one warp; a strip's column sums over all rows by one CTA, summed in
// a fixed order, so results do not depend on scheduling), and each CTA asks
// for the rows of its next product (all of them, or of large products the
// first few) to be brought into L2 before it waits at the barrier and loads
// the first part of it into registers.  A step, forward
// and backward: b = 300 9.7 and 17.3 -> 6.6 and 8.0 us, b = 1500 24.9 and 39.4
// -> 11.5 and 13.5 us (2.3 and 2.0 TB/s), against four CTAs of 8 warps per SM
// with partial column sums in global memory and none of the above.  The
// arrowhead tip is solved by the tile sweep's arrow kernels before (backward)
// or after (forward).
#include <algorithm>
#include <cstring>
#include <vector>

#include "bta_internal.cuh"
#include "common.cuh"
#include "prof.cuh"
#include "tune.cuh"

namespace bta {
namespace {

constexpr int PS_THREADS = 512;
constexpr int PS_WARPS = PS_THREADS / 32;
constexpr int PS_MAXI = 64;
constexpr int PS_COLS = 16;    // columns of a backward strip (a 128-byte segment per row)
constexpr int PS_CHUNK = 4096;  // vector entries staged at a time
constexpr double PS_BIG_BYTES = 64e6;         // of the larger product of a step: half of L2
constexpr int PS_BIG_FETCH = (12 << 20) / 8;  // entries asked for ahead of a barrier when it is larger
constexpr long long PS_SPIN_LIMIT = 1LL << 24;

struct PInst {
  const double* L;   // (n-1) b x b sub-diagonal factor blocks, or nullptr (n = 1)
  const double* Ab;  // n a x b arrow blocks, or nullptr
  const double* V;   // inverse of block vlo at V, block i at V + (i - vlo) b^2
  double* x;         // n b + a, in place
  double* t;         // b: right-hand side of a step's second product
  int n, b, a, vlo;
  int row0, pair0;   // first row, and first pair of rows, of this instance in the batch
  int strip0;        // first strip of this instance in the batch
};

struct PSweep {
  int count, trans, s0, s1;
  int units;      // rows (forward) or strips (backward) of all instances
  int pairs;      // pairs of rows of all instances
  unsigned* bar;  // arrivals
  int* abort_flag;
  PInst inst[PS_MAXI];
};

__device__ __forceinline__ unsigned ld_acquire_u(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void prefetch_l2(const double* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Grid-wide barrier of a cooperative launch (every CTA resident): arrivals
// count up for the whole launch, barrier g (from 0) is passed at (g + 1) x
// grid of them; a release-add and an acquire-poll, no further fences.  Bounded:
// a wait that runs out sets the abort flag, and every later barrier gives up
// after a few polls, so the launch always ends.  Returns false once aborted.
__device__ __forceinline__ bool grid_barrier(const PSweep& P, unsigned& gen) {
  __shared__ int s_ok;
  __syncthreads();
  ++gen;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(P.bar) : "memory");
    const unsigned target = gen * gridDim.x;
    int ok = 1;
    for (long long it = 0; (int)(ld_acquire_u(P.bar) - target) < 0; ++it) {
      if ((it & 15) == 15 && ld_acquire(P.abort_flag)) {
        ok = 0;
        break;
      }
      if (it > PS_SPIN_LIMIT) {
        atomicExch(P.abort_flag, 1);
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// v[0 .. cnt) into smem (written by other CTAs of this launch: from L2)
__device__ __forceinline__ void stage(double* sv, const double* v, int cnt) {
  for (int k = threadIdx.x; k < cnt; k += PS_THREADS) sv[k] = __ldcg(v + k);
}

// The first entries of a warp's row, or of a thread's column segment, of the
// product that follows a barrier: loaded before it (the blocks are read-only),
// so that their latency runs beside the barrier's.  at: what they are of.
constexpr int PS_PRE = 8;  // 16-byte pairs per lane, or entries per thread
struct PreRow {
  const double* at = nullptr;
  double2 m[PS_PRE];
};
struct PreStrip {
  const double* at = nullptr;
  double m[2 * PS_PRE];
};

__device__ __forceinline__ int head_of(const double* M) { return (int)(reinterpret_cast<uintptr_t>(M) >> 3) & 1; }

__device__ __forceinline__ void load_pairs(const double* M, int cnt, int q, double2 (&m)[PS_PRE]) {
  const int head = head_of(M), pairs = cnt > head ? (cnt - head) >> 1 : 0;
  const double2* m2 = reinterpret_cast<const double2*>(M + head);
#pragma unroll
  for (int j = 0; j < PS_PRE; ++j) m[j] = q + 32 * j < pairs ? __ldg(m2 + q + 32 * j) : make_double2(0.0, 0.0);
}

// Dot product of cnt entries at M with sv, by one warp.  M may start between
// two 16-byte boundaries: the first entry is then taken apart.
__device__ __forceinline__ double warp_dot(const double* M, const double* sv, int cnt, int lane, const PreRow& pre) {
  double s0 = 0.0, s1 = 0.0;
  const int head = head_of(M);
  if (head && cnt > 0 && lane == 0) s0 = __ldg(M) * sv[0];
  const double* w = sv + head;
  const int pairs = cnt > head ? (cnt - head) >> 1 : 0;
  for (int q = lane; q - lane < pairs; q += 32 * PS_PRE) {  // PS_PRE loads in flight
    double2 m[PS_PRE];
    if (q == lane && pre.at == M) {
#pragma unroll
      for (int j = 0; j < PS_PRE; ++j) m[j] = pre.m[j];
    } else {
      load_pairs(M, cnt, q, m);
    }
#pragma unroll
    for (int j = 0; j < PS_PRE; ++j)
      if (q + 32 * j < pairs) {
        s0 = fma(m[j].x, w[2 * (q + 32 * j)], s0);
        s1 = fma(m[j].y, w[2 * (q + 32 * j) + 1], s1);
      }
  }
  if (cnt > head && ((cnt - head) & 1) && lane == 0) s1 = fma(__ldg(M + cnt - 1), sv[cnt - 1], s1);
  double s = s0 + s1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Rows of a CTA that are not contiguous: those numbered mid and up lie skip
// rows further down.
struct Gap {
  int mid, skip;
};
template <bool GAP>
__device__ __forceinline__ int row_of(int q, Gap gap) {
  return GAP && q >= gap.mid ? q + gap.skip : q;
}

// out[r] = (in ? in[r] : 0) + sign sum_{k < len(r)} M[r][k] v[k] for rows
// [r0, r1), len(r) = r + 1 for a lower-triangular M, else b.
template <bool GAP = false>
__device__ __forceinline__ void rows_product(const double* M, int b, int r0, int r1, bool tri, const double* v,
                                             const double* in, double sign, double* out, double* sv,
                                             const PreRow& pre, Gap gap = Gap()) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool once = b <= PS_CHUNK;  // the whole vector stays staged
  __syncthreads();                  // the previous product's reads of sv
  if (once) {
    stage(sv, v, tri ? row_of<GAP>(r1 - 1, gap) + 1 : b);
    __syncthreads();
  }
  for (int rb = r0; rb < r1; rb += PS_WARPS) {
    const int q = rb + warp, r = row_of<GAP>(q, gap);
    const int len = q < r1 ? (tri ? r + 1 : b) : 0;
    double s = 0.0;
    if (once) {
      s = warp_dot(M + (size_t)r * b, sv, len, lane, pre);
    } else {
      const int top = tri ? row_of<GAP>(min(r1, rb + PS_WARPS) - 1, gap) + 1 : b;
      for (int k0 = 0; k0 < top; k0 += PS_CHUNK) {
        __syncthreads();
        stage(sv, v + k0, min(PS_CHUNK, top - k0));
        __syncthreads();
        // a preloaded row is one of at most PS_CHUNK entries
        s += warp_dot(M + (size_t)r * b + k0, sv, max(0, min(PS_CHUNK, len - k0)), lane, PreRow());
      }
    }
    if (lane == 0 && q < r1) out[r] = (in ? __ldcg(in + r) : 0.0) + sign * s;
  }
}

template <bool GAP = false>
__device__ __forceinline__ void preload_row(const double* M, int b, int r0, int r1, bool tri, PreRow& pre,
                                            Gap gap = Gap()) {
  const int q = r0 + (threadIdx.x >> 5), r = row_of<GAP>(q, gap);
  pre.at = nullptr;
  if (b > PS_CHUNK || q >= r1) return;
  pre.at = M + (size_t)r * b;
  load_pairs(pre.at, tri ? r + 1 : b, threadIdx.x & 31, pre.m);
}

// Rows r, r + 32, ... below k1 of a column.
__device__ __forceinline__ void load_column(const double* col, int b, int r, int k1, double (&m)[2 * PS_PRE]) {
#pragma unroll
  for (int j = 0; j < 2 * PS_PRE; ++j) m[j] = r + 32 * j < k1 ? __ldg(col + (size_t)(r + 32 * j) * b) : 0.0;
}

// Columns c0 .. c0 + 15 of M^T v over rows [rlo, b) (and of A^T va over the a
// rows of A), out[c] = (in ? in[c] : 0) + sign sum.  Each half-warp takes every
// 32nd row; the 32 sums of a column meet in shared memory.
__device__ __forceinline__ void strip_product(const double* M, int b, int c0, int rlo, const double* v,
                                              const double* A, int a, const double* va, const double* in,
                                              double sign, double* out, double* sv, double (*red)[PS_COLS],
                                              bool staged, const PreStrip& pre) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = c0 + (lane & (PS_COLS - 1)), grp = 2 * warp + (lane >> 4);
  const bool ok = c < b;
  double acc = 0.0;
  if (M != nullptr) {
    const double* col = M + c;
    for (int k0 = 0; k0 < b; k0 += PS_CHUNK) {
      const int k1 = min(b, k0 + PS_CHUNK);
      if (!staged) {
        __syncthreads();
        stage(sv, v + k0, k1 - k0);
        __syncthreads();
      }
      if (ok)
        for (int r = max(k0, rlo) + grp; r < k1; r += 64 * PS_PRE) {  // 2 PS_PRE loads in flight
          double m[2 * PS_PRE];
          if (pre.at == col && r == rlo + grp) {
#pragma unroll
            for (int j = 0; j < 2 * PS_PRE; ++j) m[j] = pre.m[j];
          } else {
            load_column(col, b, r, k1, m);
          }
#pragma unroll
          for (int j = 0; j < 2 * PS_PRE; ++j)
            if (r + 32 * j < k1) acc = fma(m[j], sv[r + 32 * j - k0], acc);
        }
    }
  }
  if (ok)
    for (int q = grp; q < a; q += 32) acc = fma(__ldg(A + (size_t)q * b + c), __ldcg(va + q), acc);
  acc += __shfl_xor_sync(0xffffffffu, acc, 16);
  __syncthreads();  // red of the previous strip
  if (lane < PS_COLS) red[warp][lane] = acc;
  __syncthreads();
  if (warp == 0) {
    const int cc = lane & (PS_COLS - 1), h = lane >> 4;
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < PS_WARPS / 2; ++w) s += red[h * (PS_WARPS / 2) + w][cc];
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    if (lane < PS_COLS && c0 + cc < b) out[c0 + cc] = (in ? __ldcg(in + c0 + cc) : 0.0) + sign * s;
  }
}

// The rows that strip_product takes first: from rlo on, to the end of the
// staged chunk that holds row rlo.
__device__ __forceinline__ void preload_strip(const double* M, int b, int c0, int rlo, PreStrip& pre) {
  const int lane = threadIdx.x & 31, c = c0 + (lane & (PS_COLS - 1));
  pre.at = nullptr;
  if (c >= b) return;
  pre.at = M + c;
  load_column(pre.at, b, rlo + 2 * (threadIdx.x >> 5) + (lane >> 4), min(b, (rlo / PS_CHUNK + 1) * PS_CHUNK), pre.m);
}

// BIG: a step's larger product has more than PS_BIG_BYTES.  Asking for all of
// the next product then drives lines out of L2 before they are used, so a CTA
// asks for PS_BIG_FETCH / grid entries ahead of a barrier only, about what
// memory delivers during the barrier (8 to 32 MB measured alike).  Such steps
// are bound by bandwidth, so the forward sweep's triangular product is split
// by pairs of rows q and b - 1 - q: contiguous rows give the last CTA of a
// block twice the average.  Forward and backward, all asked for against BIG:
// 12 x 20 blocks of 1500 (216 MB) 2.14 and 2.28 -> 1.58 and 1.83 ms, 6 x 100
// of 1500 (108 MB) 4.98 and 5.52 -> 4.06 and 4.82, 20 of 4000 (128 MB) 1.07 and
// 1.22 -> 0.77 and 1.05.  Below the line all is better: 60 of 2500 (50 MB)
// 1.52 and 2.06 against 1.38 and 2.11, 16 x 40 of 600 (46 MB) 1.32 and 1.42
// against 1.34 and 1.46, 16 of 1117 (10 MB) 0.158 and 0.194 against 0.167 and
// 0.198 ms.
template <bool BIG>
__global__ void __launch_bounds__(PS_THREADS) sweep_persist_kernel(const __grid_constant__ PSweep P) {
  __shared__ __align__(16) double sv[PS_CHUNK];
  __shared__ double red[PS_WARPS][PS_COLS];
  unsigned gen = 0;
  // this CTA's share of the rows or strips
  const int u0 = (int)((long long)P.units * blockIdx.x / gridDim.x);
  const int u1 = (int)((long long)P.units * (blockIdx.x + 1) / gridDim.x);
  // f(instance, first, last): this CTA's share of each instance
  auto each = [&](auto f) {
    for (int k = 0; k < P.count; ++k) {
      const PInst& I = P.inst[k];
      const int lo = P.trans == 0 ? I.row0 : I.strip0;
      if (BIG && lo >= u1) break;
      const int cnt = P.trans == 0 ? I.b : (I.b + PS_COLS - 1) / PS_COLS;
      const int a = max(u0, lo), e = min(u1, lo + cnt);
      if (a < e) f(I, a - lo, e - lo);
    }
  };
  // the first instance of this CTA's share: its first product after a barrier
  // is preloaded
  int kf = 0;
  while (kf + 1 < P.count && u0 >= (P.trans == 0 ? P.inst[kf + 1].row0 : P.inst[kf + 1].strip0)) ++kf;
  const PInst& F = P.inst[kf];
  const int f0 = u0 - (P.trans == 0 ? F.row0 : F.strip0);
  const int f1 = min(u1 - (P.trans == 0 ? F.row0 : F.strip0), P.trans == 0 ? F.b : (F.b + PS_COLS - 1) / PS_COLS);
  const size_t fbb = (size_t)F.b * F.b;
  // lines of rows [r0, r1) of a b-wide block, or of 16-column strips [s0, s1)
  // of its rows from rlo on
  const int room = PS_BIG_FETCH / (int)gridDim.x;
  int left = room;
  // m of the units of `per` entries each that may still be asked for
  auto take = [&](int m, int per) {
    if constexpr (BIG) {
      m = min(m, left / per);
      left -= m * per;
    }
    return m;
  };
  auto fetch_rows = [&](const double* M, int b, int r0, int r1) {
    const size_t e0 = (size_t)r0 * b, e1 = (size_t)(r0 + take(r1 - r0, b)) * b;
    for (size_t e = e0 + 16 * threadIdx.x; e < e1; e += 16 * PS_THREADS) prefetch_l2(M + e);
  };
  auto fetch_tri = [&](const double* M, int b, int r0, int r1, Gap gap) {
    const int e1 = r0 + take(r1 - r0, (b + 1) / 2);
    for (int q = r0 + (threadIdx.x >> 5); q < e1; q += PS_WARPS)
      for (int r = row_of<BIG>(q, gap), k = 16 * (threadIdx.x & 31); k <= r; k += 512)
        prefetch_l2(M + (size_t)r * b + k);
  };
  auto fetch_strips = [&](const double* M, int b, int s0, int s1, bool tri) {
    const int rlo = tri ? PS_COLS * s0 : 0, w = take(s1 - s0, PS_COLS * (b - rlo));
    for (int q = threadIdx.x; q < (b - rlo) * w; q += PS_THREADS)
      prefetch_l2(M + (size_t)(rlo + q / w) * b + PS_COLS * (s0 + q % w));
  };
  // f(instance, first, last, gap): this CTA's rows of the forward sweep's
  // triangular products; BIG: pairs [a, e) of an instance, which are its rows
  // [a, e) and [b - e, b - a) (the middle row of an odd b once)
  auto each_tri = [&](auto f) {
    if constexpr (BIG) {
      const int q0 = (int)((long long)P.pairs * blockIdx.x / gridDim.x);
      const int q1 = (int)((long long)P.pairs * (blockIdx.x + 1) / gridDim.x);
      for (int k = 0; k < P.count && P.inst[k].pair0 < q1; ++k) {
        const PInst& I = P.inst[k];
        const int a = max(q0 - I.pair0, 0), e = min(q1 - I.pair0, (I.b + 1) / 2), hi = max(I.b - e, e);
        if (a < e) f(I, a, e + I.b - a - hi, Gap{e, hi - e});
      }
    } else {
      each([&](const PInst& I, int r0, int r1) { f(I, r0, r1, Gap()); });
    }
  };

  if (P.trans == 0) {
    PreRow pre;
    if (P.s0 > 0 && P.s0 < F.n) preload_row(F.L + (P.s0 - 1) * fbb, F.b, f0, f1, false, pre);
    for (int st = P.s0; st < P.s1; ++st) {
      left = room;
      each([&](const PInst& I, int r0, int r1) {
        if (st >= I.n) return;
        double* xi = I.x + (size_t)st * I.b;
        if (st > 0) {
          // t = b_i - L_{i,i-1} y_{i-1}
          rows_product(I.L + (size_t)(st - 1) * I.b * I.b, I.b, r0, r1, false, xi - I.b, xi, -1.0, I.t, sv, pre);
        } else {
          for (int r = r0 + threadIdx.x; r < r1; r += PS_THREADS) I.t[r] = __ldcg(xi + r);
        }
        if constexpr (!BIG) fetch_tri(I.V + (size_t)(st - I.vlo) * I.b * I.b, I.b, r0, r1, Gap());
      });
      pre.at = nullptr;
      if constexpr (BIG) {
        bool first = true;
        each_tri([&](const PInst& I, int r0, int r1, Gap gap) {
          const double* Vi = I.V + (size_t)(st - I.vlo) * I.b * I.b;
          if (st < I.n) fetch_tri(Vi, I.b, r0, r1, gap);
          if (st < I.n && first) preload_row<true>(Vi, I.b, r0, r1, true, pre, gap);
          first = false;
        });
      } else if (st < F.n) {
        preload_row(F.V + (st - F.vlo) * fbb, F.b, f0, f1, true, pre);
      }
      if (!grid_barrier(P, gen)) return;
      left = room;
      each_tri([&](const PInst& I, int r0, int r1, Gap gap) {
        if (st >= I.n) return;
        // y_i = V_i t
        rows_product<BIG>(I.V + (size_t)(st - I.vlo) * I.b * I.b, I.b, r0, r1, true, I.t, nullptr, 1.0,
                          I.x + (size_t)st * I.b, sv, pre, gap);
        if constexpr (!BIG)
          if (st + 1 < min(P.s1, I.n)) fetch_rows(I.L + (size_t)st * I.b * I.b, I.b, r0, r1);
      });
      if constexpr (BIG)
        each([&](const PInst& I, int r0, int r1) {
          if (st + 1 < min(P.s1, I.n)) fetch_rows(I.L + (size_t)st * I.b * I.b, I.b, r0, r1);
        });
      pre.at = nullptr;
      if (st + 1 < min(P.s1, F.n)) preload_row(F.L + st * fbb, F.b, f0, f1, false, pre);
      if (!grid_barrier(P, gen)) return;
    }
    return;
  }

  // backward: step st handles block i = n - 1 - st of every instance
  PreStrip pre;
  {
    const int i = F.n - 1 - P.s0;
    if (i >= 0 && i < F.n - 1) preload_strip(F.L + i * fbb, F.b, PS_COLS * f0, 0, pre);
  }
  for (int st = P.s0; st < P.s1; ++st) {
    const int fi = F.n - 1 - st;  // the first instance's block
    left = room;
    each([&](const PInst& I, int s0, int s1) {
      const int i = I.n - 1 - st;
      if (i < 0) return;
      // t = y_i - L_i^T x_{i+1} - Ab_i^T x_a
      double* xi = I.x + (size_t)i * I.b;
      const double* Li = i < I.n - 1 ? I.L + (size_t)i * I.b * I.b : nullptr;
      const double* Ai = I.a > 0 ? I.Ab + (size_t)i * I.a * I.b : nullptr;
      const bool once = I.b <= PS_CHUNK;
      if (once && Li) {
        __syncthreads();
        stage(sv, xi + I.b, I.b);
        __syncthreads();
      }
      for (int s = s0; s < s1; ++s)
        strip_product(Li, I.b, PS_COLS * s, 0, xi + I.b, Ai, I.a, I.x + (size_t)I.n * I.b, xi, -1.0, I.t, sv, red, once,
                      pre);
      fetch_strips(I.V + (size_t)(i - I.vlo) * I.b * I.b, I.b, s0, s1, true);
    });
    pre.at = nullptr;
    if (fi >= 0) preload_strip(F.V + (fi - F.vlo) * fbb, F.b, PS_COLS * f0, PS_COLS * f0, pre);
    if (!grid_barrier(P, gen)) return;
    left = room;
    each([&](const PInst& I, int s0, int s1) {
      const int i = I.n - 1 - st;
      if (i < 0) return;
      // x_i = V_i^T t
      const bool once = I.b <= PS_CHUNK;
      if (once) {
        __syncthreads();
        stage(sv, I.t, I.b);
        __syncthreads();
      }
      for (int s = s0; s < s1; ++s)
        strip_product(I.V + (size_t)(i - I.vlo) * I.b * I.b, I.b, PS_COLS * s, PS_COLS * s, I.t, nullptr, 0, nullptr,
                      nullptr, 1.0, I.x + (size_t)i * I.b, sv, red, once, pre);
      if (i > 0 && st + 1 < P.s1) fetch_strips(I.L + (size_t)(i - 1) * I.b * I.b, I.b, s0, s1, false);
    });
    pre.at = nullptr;
    if (fi > 0 && st + 1 < P.s1) preload_strip(F.L + (fi - 1) * fbb, F.b, PS_COLS * f0, 0, pre);
    if (!grid_barrier(P, gen)) return;
  }
}

}  // namespace

size_t sweep_inv_work(int n, int b, int a) { return (size_t)b + (size_t)n * a + 64; }

int sweep_inv_steps(int count, const int* n, const int* b, const int* a, const double* const* L,
                    const double* const* Ab, const double* const* V, const int* vlo, double* const* x, int trans,
                    int s0, int s1, double* work, int* abort_flag, cudaStream_t s) {
  if (count < 1 || count > PS_MAXI || s1 <= s0) return count < 1 || count > PS_MAXI ? cudaErrorInvalidValue : 0;
  int bsum = 0, bmax = 0;
  for (int k = 0; k < count; ++k) {
    bsum += b[k];
    bmax = std::max(bmax, b[k]);
  }
  // candidates: a CTA per SM, or per two SMs (a quicker barrier, for small
  // blocks); two on an SM do not fit (512 threads of 124 registers).  Each is
  // tried twice: the first launch of a process also loads the kernel
  TuneLaunch tl("sweep", {count, trans, bsum, bmax, s1 - s0}, 2, s);
  const int cand = tl.choice();
  PSweep P;
  std::memset(&P, 0, sizeof(P));
  P.count = count;
  P.trans = trans;
  P.s0 = s0;
  P.s1 = s1;
  P.abort_flag = abort_flag;
  size_t off = 0;
  double bytes = 0;  // of the step's larger product
  for (int k = 0; k < count; ++k) {
    PInst& I = P.inst[k];
    I.L = n[k] > 1 ? L[k] : nullptr;
    I.Ab = a[k] > 0 ? Ab[k] : nullptr;
    I.V = V[k];
    I.vlo = vlo ? vlo[k] : 0;
    I.x = x[k];
    I.n = n[k];
    I.b = b[k];
    I.a = a[k];
    I.t = work + off;
    off += sweep_inv_work(n[k], b[k], a[k]);
    if (trans == 0) I.row0 = P.units;
    else I.strip0 = P.units;
    I.pair0 = P.pairs;
    P.pairs += (b[k] + 1) / 2;
    bytes += 8.0 * b[k] * b[k];
    P.units += trans == 0 ? b[k] : (b[k] + PS_COLS - 1) / PS_COLS;
  }
  // barrier words after the instances' scratch
  P.bar = reinterpret_cast<unsigned*>(work + off);
  if (cudaMemsetAsync(P.bar, 0, 2 * sizeof(unsigned), s) != cudaSuccess) return cudaErrorUnknown;
  auto kernel = bytes > PS_BIG_BYTES ? sweep_persist_kernel<true> : sweep_persist_kernel<false>;
  const int sms = device_sm_count();
  // no more CTAs than there are groups of 8 rows, or strips
  const int most = std::max(1, trans == 0 ? (P.units + 7) / 8 : P.units);
  const int grid = std::min(most, cand == 0 ? sms : std::max(1, sms / 2));
  void* args[] = {&P};
  bta::ProfScope _ps(bta::PROF_SWEEP, s);
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(grid),
                                     dim3(PS_THREADS), args, 0, s);
}

size_t sweep_inv_work_total(int count, const int* n, const int* b, const int* a) {
  size_t w = 0;
  for (int k = 0; k < count; ++k) w += sweep_inv_work(n[k], b[k], a[k]);
  return w + 64;
}

int sweep_inv_batched(int count, const int* n, const int* b, const int* a, const double* const* L,
                      const double* const* Ab, const double* const* T, const double* const* V, double* const* x,
                      int trans, double* work, int* abort_flag, cudaStream_t s) {
  int maxn = 0;
  for (int k = 0; k < count; ++k) maxn = std::max(maxn, n[k]);
  // arrow scratch of the forward arrow step after the instances' sweep scratch
  double* apart = work + sweep_inv_work_total(count, n, b, a);
  if (trans == 1)
    for (int k = 0; k < count; ++k)
      if (a[k] > 0 && arrow_backward(T[k], x[k], n[k], b[k], a[k], s)) return cudaErrorUnknown;
  for (int c0 = 0; c0 < count; c0 += PS_MAXI) {
    const int c1 = std::min(count, c0 + PS_MAXI);
    int cn = 0;
    for (int k = c0; k < c1; ++k) cn = std::max(cn, n[k]);
    const int e = sweep_inv_steps(c1 - c0, n + c0, b + c0, a + c0, L + c0, Ab + c0, V + c0, nullptr, x + c0, trans,
                                  0, cn, work, abort_flag, s);
    if (e) return e;
  }
  if (trans == 0)
    for (int k = 0; k < count; ++k) {
      if (a[k] <= 0) continue;
      if (arrow_forward(Ab[k], T[k], x[k], n[k], b[k], a[k], apart, s)) return cudaErrorUnknown;
    }
  return cudaGetLastError();
}

}  // namespace bta
