// 64x64 FP64 tile operations in shared memory, used by several kernels.
#pragma once

#include "common.cuh"

namespace bta {
namespace tile {

constexpr int T = TILE;
constexpr int THREADS = 128;
constexpr int SG = T + 4;  // stride of GEMM operand tiles (k-contiguous, conflict-free)

// Load a rows x cols tile (leading dimension ld) into smem with stride S,
// zero-filled to 64 x 64.  L2-only loads (data may come from other CTAs).
template <int S>
__device__ __forceinline__ void load(double* s, const double* g, int ld, int rows, int cols, int tid) {
#pragma unroll 8
  for (int idx = tid; idx < T * T; idx += THREADS) {
    const int r = idx >> 6, c = idx & 63;
    s[r * S + c] = (r < rows && c < cols) ? __ldcg(g + (size_t)r * ld + c) : 0.0;
  }
}

// Asynchronous version of load() for an even stride S: 16-byte cp.async
// (L2 only, zero-filled) when the tile rows are 16-byte aligned, scalar L2
// loads otherwise.  The caller commits, waits and synchronises.
template <int S>
__device__ __forceinline__ void load_async(double* s, const double* g, int ld, int rows, int cols, int tid) {
  static_assert((S & 1) == 0, "16-byte smem rows");
  const bool vec = ((ld & 1) == 0) && ((reinterpret_cast<uintptr_t>(g) & 15) == 0);
  if (vec) {
#pragma unroll
    for (int j = 0; j < (T * T / 2) / THREADS; ++j) {
      const int c = tid + j * THREADS;
      const int r = c >> 5, col = (c & 31) * 2;
      const int nvalid = (r < rows) ? max(0, min(2, cols - col)) : 0;
      const double* src = nvalid ? g + (size_t)r * ld + col : g;
      const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(s + r * S + col));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(src), "r"(nvalid * 8));
    }
  } else {
    load<S>(s, g, ld, rows, cols, tid);
  }
}

// Row blocks whose rows are not all 16-byte aligned (an odd row stride, or a
// base between two 16-byte boundaries): rows with odd parity are copied from
// the boundary before them, so that 16-byte cp.async serves them too, and lie
// one element further right in shared memory.  The parity of row r is
// row_parity(g, ld, r); a thread of an m16n8k4 product reads rows that are
// congruent to its g modulo 8 only, so its shift is one constant.
__device__ __forceinline__ int row_parity(const double* g, int ld, int r) {
  return ((int)(reinterpret_cast<uintptr_t>(g) >> 3) + (r & ld)) & 1;
}

// R rows x W columns from column k0 of a row block at g into smem rows of
// stride S (W + 2 <= S, both even), shifted by the rows' parity; rows < rows
// and columns < kmax, zeros beyond.  L2 only.  The element before an odd row
// is copied along and never read: it is in the row's first 16-byte granule.
template <int R, int W, int S>
__device__ __forceinline__ void load_shifted_async(double* s, const double* g, int ld, int rows, int k0, int kmax,
                                                   int tid) {
  static_assert(W + 2 <= S && (S & 1) == 0, "shifted rows overlap");
  constexpr int NC = W / 2, RS = THREADS / NC;  // whole chunks of a row, rows per pass
  static_assert(RS % 2 == 0, "a thread's rows have one parity");
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(s));
  auto copy = [&](int r, int c, int par) {
    const int e = k0 + 2 * c - par;
    const int nvalid = r < rows ? max(0, min(2, kmax - e)) : 0;
    const double* src = nvalid ? g + ((size_t)r * ld + e) : g + row_parity(g, ld, 0);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa + (r * S + 2 * c) * 8), "l"(src),
                 "r"(nvalid * 8));
  };
  const int r0 = tid / NC, c0 = tid % NC, par0 = row_parity(g, ld, r0);
#pragma unroll
  for (int j = 0; j < R / RS; ++j) copy(r0 + RS * j, c0, par0);
  // the last element of an odd row
  if (tid < R && row_parity(g, ld, tid)) copy(tid, NC, 1);
}

__device__ __forceinline__ void zero_acc(double (&acc)[2][4][4]) {
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[mi][ni][e] = 0.0;
}

// acc[n] += rows 16 warp .. of X times columns 8 n .. of Y^T for a lower
// triangular Y (both k-contiguous, stride SG): column n sums k <= n only, so
// the 16x8 tile n runs 2 (n + 1) of 16 k-steps and, a warp owning 16 whole
// rows, the four warps have the same work (72 products each; with a 32x32
// quarter per warp two of them had 128).  Y's 8x8 diagonal blocks hold zeros
// above the diagonal.  shift: of this thread's rows of X (row_parity).
__device__ __forceinline__ void tri_mma_nt(const double* X, const double* Y, double (&acc)[8][4], int warp, int g,
                                           int t, int shift = 0) {
  const double* x = X + (16 * warp + g) * SG + t + shift;
  const double* y = Y + g * SG + t;
#pragma unroll
  for (int kk = 0; kk < T; kk += 4) {
    const double a0 = x[kk], a1 = x[8 * SG + kk];
#pragma unroll
    for (int n = kk / 8; n < 8; ++n) dmma16x8x4(acc[n], a0, a1, y[8 * n * SG + kk]);
  }
}

// 1/sqrt(x) for x > 0: hardware seed (rsqrt.approx, within 1e-6) and one
// cubic correction, y <- y (1 + r/2 + 3 r^2/8) with r = 1 - x y^2 (the series
// of (1 - r)^{-1/2}): four dependent operations, against nine of three Newton
// steps.  Within 1.5 x 2^-53 of 1/sqrt(x) for normal x: the rounding of x y,
// half of which r carries over, and that of the result.
__device__ __forceinline__ double rsqrt_cubic(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double r = fma(-x * y, y, 1.0);
  return fma(y * r, fma(0.375, r, 0.5), y);
}

// 1/x: hardware seed refined by Newton-Raphson for 1/x, y <- y + y (1 - x y).
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#pragma unroll
  for (int it = 0; it < 3; ++it) {
    const double r = fma(-x, y, 1.0);
    y = fma(y, r, y);
  }
  return y;
}

// Rows below 16-wide panel KB of potrf_inv: S -= X X^T (lower 16x8 tiles),
// V -= X V_panel, with X = S[rows below][panel].  A tile's operands are
// loaded while the previous tile's products run.
template <int KB>
__device__ __forceinline__ void potrf_inv_trailing(double* S, double* V, int warp, int g, int t) {
  constexpr int o = KB * 16, mt = 3 - KB, na = mt * (mt + 1), nv = 2 * (KB + 1), ntile = na + mt * nv;
  constexpr int NU = (ntile + 3) / 4;
  double a[2][8], b[2][4];
  const int gt = g * SG + t;
  // tile u of the warp: row tile mi; column tile ni of S, or of V when ni >= 8
  auto place = [&](int u, int& mi, int& ni) {
    const int tile = warp + 4 * u, v = tile - na;
    if (tile < na) {
      mi = tile < 2 ? 0 : tile < 6 ? 1 : 2;
      ni = tile - mi * (mi + 1);
    } else {
      mi = v / nv;
      ni = 8 + v - mi * nv;
    }
  };
  auto load = [&](int u, double (&ra)[8], double (&rb)[4]) {
    int mi, ni;
    place(u, mi, ni);
    const double* A = S + (o + 16 + mi * 16) * SG + o + gt;
    const double* B = ni < 8 ? S + (o + 16 + ni * 8) * SG + o + gt : V + o * SG + (ni - 8) * 8 + t * SG + g;
    const int bs = ni < 8 ? 1 : SG;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      ra[2 * k] = -A[4 * k];
      ra[2 * k + 1] = -A[8 * SG + 4 * k];
      rb[k] = B[4 * k * bs];
    }
  };
  load(0, a[0], b[0]);
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    if (warp + 4 * u >= ntile) break;
    int mi, ni;
    place(u, mi, ni);
    double* C = (ni < 8 ? S + o + 16 + ni * 8 : V + (ni - 8) * 8) + (o + 16 + mi * 16 + g) * SG + 2 * t;
    double2 c0 = make_double2(0.0, 0.0), c1 = c0;
    if (ni < 8 + 2 * KB) {  // the panel's own columns of V start at zero
      c0 = *reinterpret_cast<double2*>(C);
      c1 = *reinterpret_cast<double2*>(C + 8 * SG);
    }
    if (u + 1 < NU) load(min(u + 1, (ntile - 1 - warp) / 4), a[(u + 1) & 1], b[(u + 1) & 1]);
    double acc[4] = {c0.x, c0.y, c1.x, c1.y};
#pragma unroll
    for (int k = 0; k < 4; ++k) dmma16x8x4(acc, a[u & 1][2 * k], a[u & 1][2 * k + 1], b[u & 1][k]);
    *reinterpret_cast<double2*>(C) = make_double2(acc[0], acc[1]);
    *reinterpret_cast<double2*>(C + 8 * SG) = make_double2(acc[2], acc[3]);
  }
}

// In-place lower Cholesky of the 64x64 smem tile S and the inverse of its
// factor in V (both stride SG), in 16-wide panels.  Rows and columns from w
// to the end of their panel are treated as the identity, panels beyond are
// left out (some 3.6 k cycles each).  A
// non-positive pivot j < w records base+j+1 in *info (atomicMin); the
// factorisation continues.  On exit the lower triangles of S and V hold L and
// L^-1 in the rows of those panels, their 16x16 diagonal blocks zeros above
// the diagonal; the blocks above those and the rows after them hold nothing
// of use.
// The caller synchronises before (S complete) and needs no barrier after.
//
// The chain of 64 dependent pivots bounds this routine, so nothing else is
// serial: every warp runs a panel's 16 pivots on the panel's diagonal block
// (lanes 0-15, one row each, the same in all warps) and, in the same
// instructions, on 16 other rows (lanes 16-31) -- rows of S below the block,
// whose triangular solve thereby costs nothing, or columns of the inverse,
// because V satisfies the recurrence of a row below with the identity as its
// input (48 - 16 kb rows and 16 (kb + 1) columns: 64 in every panel).  A
// pivot is shuffled before the other columns' updates are, so they wait in
// its shadow.  Measured on one CTA alone: 14.1 k cycles for both, against
// 24.4 k for a factorisation with a separate solve of the rows below and
// inversion afterwards.
__device__ __forceinline__ void potrf_inv(double* S, double* V, int w, unsigned long long* info, long long base,
                                          int tid) {
  // opaque: in a caller's loop the tile offsets below would be hoisted out of
  // it, into more registers than there are
  asm volatile("" : "+r"(tid));
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int hi = lane >> 4, li = lane & 15;
  // panels beyond w are left out, rows up to the last panel's end are those
  // of the identity (what lies above the diagonal is never used)
  const int np = (w + 15) >> 4;
  if (w < 16 * np) {
    for (int idx = w * T + tid; idx < 16 * np * T; idx += THREADS) {
      const int i = idx >> 6, k = idx & 63;
      S[i * SG + k] = (i == k) ? 1.0 : 0.0;
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int kb = 0; kb < np; ++kb) {
    const int o = kb * 16;
    const int vg = warp - (3 - kb);  // >= 0: column group of V, else a group of rows below
    double d[16];
    double* src;
    if (!hi || vg < 0) {
      src = S + (o + (hi ? 16 + 16 * warp : 0) + li) * SG + o;
#pragma unroll
      for (int k = 0; k < 16; k += 2) {
        const double2 v = *reinterpret_cast<const double2*>(src + k);
        d[k] = v.x;
        d[k + 1] = v.y;
      }
    } else {
      src = V + o * SG + 16 * vg + li;
#pragma unroll
      for (int k = 0; k < 16; ++k) d[k] = warp == 3 ? (k == li ? 1.0 : 0.0) : src[k * SG];
    }
    __syncthreads();
    bool bad = false;
    int badj = 0;
    double piv = __shfl_sync(0xffffffffu, d[0], 0);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (!(piv > 0.0) && o + j < w && !bad) { bad = true; badj = o + j; }
      const double rs = rsqrt_cubic(piv);
      const double l = d[j] * rs;
      if (j + 1 < 16) {
        const double dn = fma(-l, l, d[j + 1]);
        piv = __shfl_sync(0xffffffffu, dn, j + 1);
      }
#pragma unroll
      for (int k = j + 1; k < 16; ++k) {
        const double lkj = __shfl_sync(0xffffffffu, l, k);
        d[k] = fma(-l, lkj, d[k]);
      }
      d[j] = (hi || li >= j) ? l : 0.0;
    }
    if (bad && tid == 0 && info != nullptr) atomicMin(info, (unsigned long long)(base + badj + 1));
    if (vg < 0 || !hi) {
      if (hi || warp == 0) {
#pragma unroll
        for (int k = 0; k < 16; k += 2) *reinterpret_cast<double2*>(src + k) = make_double2(d[k], d[k + 1]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k) src[k * SG] = d[k];
    }
    __syncthreads();
    if (kb + 1 == np) break;
    if (kb == 0) potrf_inv_trailing<0>(S, V, warp, g, t);
    else if (kb == 1) potrf_inv_trailing<1>(S, V, warp, g, t);
    else potrf_inv_trailing<2>(S, V, warp, g, t);
    __syncthreads();
  }
}

// Li <- inverse of the lower-triangular 64x64 smem tile S (both stride SG;
// non-zero diagonal over the full tile).  Each warp inverts one 16x16
// diagonal block (one column per lane, substitution in registers), then the
// off-diagonal blocks follow from X21 = -inv(L22) L21 inv(L11) for h = 16, 32
// on the DMMA pipe.  rd: 64 doubles of smem scratch.
__device__ __forceinline__ void trinv(const double* S, double* Li, double* rd, int tid) {
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  for (int idx = tid; idx < T * T; idx += THREADS) Li[(idx >> 6) * SG + (idx & 63)] = 0.0;
  if (tid < T) rd[tid] = rcp_nr(S[tid * SG + tid]);
  __syncthreads();
  {
    const int o = warp * 16, c = lane & 15;
    double wv[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      double s = (i == c) ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < i; ++k) s = fma(-S[(o + i) * SG + o + k], wv[k], s);
      wv[i] = (i >= c) ? s * rd[o + i] : 0.0;
    }
    if (lane < 16) {
#pragma unroll
      for (int i = 0; i < 16; ++i) Li[(o + i) * SG + o + c] = wv[i];
    }
  }
  __syncthreads();
  for (int h = 16; h <= 32; h *= 2) {
    // unit of work: one 16x8 output tile (m16n8) of an h x h product
    const int nblk = T / (2 * h);
    const int units = nblk * (h / 16) * (h / 8);
    // Tmp = L21 * inv(L11) -> scratch in the zero upper block Li[o.., o+h..]
    for (int u = warp; u < units; u += 4) {
      const int bb = u / ((h / 16) * (h / 8)), rem = u % ((h / 16) * (h / 8));
      const int mi = rem / (h / 8), ni = rem % (h / 8), o = bb * 2 * h;
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      for (int kk = 0; kk < h; kk += 4) {
        const double a0 = S[(o + h + mi * 16 + g) * SG + o + kk + t];
        const double a1 = S[(o + h + mi * 16 + g + 8) * SG + o + kk + t];
        const double b0 = Li[(o + kk + t) * SG + o + ni * 8 + g];
        dmma16x8x4(acc, a0, a1, b0);
      }
      double* dst = Li + (o + mi * 16 + g) * SG + o + h + ni * 8 + 2 * t;
      dst[0] = acc[0];
      dst[1] = acc[1];
      dst[8 * SG] = acc[2];
      dst[8 * SG + 1] = acc[3];
    }
    __syncthreads();
    // X21 = -inv(L22) * Tmp
    for (int u = warp; u < units; u += 4) {
      const int bb = u / ((h / 16) * (h / 8)), rem = u % ((h / 16) * (h / 8));
      const int mi = rem / (h / 8), ni = rem % (h / 8), o = bb * 2 * h;
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      for (int kk = 0; kk < h; kk += 4) {
        const double a0 = Li[(o + h + mi * 16 + g) * SG + o + h + kk + t];
        const double a1 = Li[(o + h + mi * 16 + g + 8) * SG + o + h + kk + t];
        const double b0 = Li[(o + kk + t) * SG + o + h + ni * 8 + g];
        dmma16x8x4(acc, a0, a1, b0);
      }
      double* dst = Li + (o + h + mi * 16 + g) * SG + o + ni * 8 + 2 * t;
      dst[0] = -acc[0];
      dst[1] = -acc[1];
      dst[8 * SG] = -acc[2];
      dst[8 * SG + 1] = -acc[3];
    }
    __syncthreads();
    for (int idx = tid; idx < nblk * h * h; idx += THREADS) {
      const int bb = idx / (h * h), rem = idx % (h * h);
      const int i = rem / h, c = rem % h, o = bb * 2 * h;
      Li[(o + i) * SG + o + h + c] = 0.0;
    }
    __syncthreads();
  }
}

}  // namespace tile
}  // namespace bta
