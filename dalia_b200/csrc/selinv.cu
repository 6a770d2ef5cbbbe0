// Full inverses of the diagonal factor blocks (used by the selected inversion)
// and the deterministic log-determinant reduction.
#include <algorithm>
#include <cstring>

#include "bta_internal.cuh"
#include "common.cuh"
#include "tile_ops.cuh"
#include "prof.cuh"

namespace bta {
namespace {

using namespace tile;
// Slab ring of a tile's sum: A = 64 rows x 16 k of a row block of the factor
// (k-contiguous, stride TSK), B = 16 k x 64 columns of the output
// (n-contiguous, stride TSN), two stages; three CTAs per SM hide the rest.
constexpr int TK = 16, TSK = TK + 4, TSN = T + 4, TST = 2;
constexpr int TA_SLAB = T * TSK, TB_SLAB = TK * TSN;
// shared memory: the ring (also the staging of a tile's sum, 64 x SG), then
// the diagonal tile inverse (64 x SG)
constexpr int TRTRI_RING = TST * (TA_SLAB + TB_SLAB) > T * SG ? TST * (TA_SLAB + TB_SLAB) : T * SG;
constexpr int TRTRI_CTAS = 3;  // per SM, by registers and shared memory
constexpr size_t TRTRI_SMEM = size_t(TRTRI_RING + T * SG) * sizeof(double);

// One instance of a launch: n lower-triangular blocks of b x b at D, their
// inverses to out.
struct TrtriDev {
  const double* D;
  double* out;
  long long flag0;  // first flag: [block][tile column][tile row]
  int n, b, nq;
};

constexpr int TRTRI_MAXI = 64;
constexpr double COLUMN_WORK = 0.72;  // block_trtri

struct TrtriBatch {
  int count, total;
  int zeros;     // tasks of diagonal tiles clear the column above
  int nqmax;     // largest nq
  int* flags;    // tile (p, c) of a block written
  int* counter;  // next task
  int* abort_flag;
  TrtriDev inst[TRTRI_MAXI];
};

template <bool VEC>
__device__ __forceinline__ void trtri_load(double* As, double* Bs, const double* Arow, int rows, const double* Bcol,
                                           int cols, int k0, int kend, int ld, int tid) {
  if constexpr (!VEC) {
    load_shifted_async<T, TK, TSK>(As, Arow, ld, rows, k0, kend, tid);
    load_shifted_async<TK, T, TSN>(Bs, Bcol + (size_t)k0 * ld, ld, kend - k0, 0, cols, tid);
    return;
  }
#pragma unroll
  for (int j = 0; j < (T * TK / 2) / THREADS; ++j) {
    const int q = tid + j * THREADS;
    // A: row r, k pair kc (kend - k0 is a multiple of 16); B: k row kr, column pair nc
    const int r = q >> 3, kc = (q & 7) * 2, kr = q >> 5, nc = (q & 31) * 2;
    cp_async16(As + r * TSK + kc, r < rows ? Arow + (size_t)r * ld + k0 + kc : Arow, r < rows);
    cp_async16(Bs + kr * TSN + nc, nc < cols ? Bcol + (size_t)(k0 + kr) * ld + nc : Bcol, nc < cols);
  }
}

// acc += A[:, k0:kend] B[k0:kend, :] with A = rows x (.) at Arow, B = (.) x cols
// at Bcol (both row stride ld), through a cp.async ring; the 64 rows of B
// from row 64 k on are read once gate[k] is set.  Returns false when a wait
// gave up.  VEC: every row is 16-byte aligned.  own: all rows of B are there (a
// run-time value also where it is always true: the loop compiled without its
// test of the gates took 3 to 6 % longer).
template <bool VEC>
__device__ __forceinline__ bool trtri_stream(const double* Arow, int rows, const double* Bcol, int cols, int k0,
                                             int kend, int ld, bool own, const int* gate, int* abort_flag, int* s_flag,
                                             double* smem, double (&acc)[2][4][4], int tid, int wm, int wn, int g,
                                             int t) {
  double* As = smem;
  double* Bs = smem + TST * TA_SLAB;
  const int sha = VEC ? 0 : row_parity(Arow, ld, g), shb = VEC ? 0 : row_parity(Bcol, ld, t);
  const int nslab = (kend - k0) / TK;
  // the leading rows already written: one scan of their flags (relaxed loads
  // in flight together, one fence), later ones are waited for one by one
  if (tid == 0 && !own) {
    int k = k0 / T;
    while (k < kend / T && ld_relaxed(gate + k) >= 1) ++k;
    __threadfence();
    s_flag[1] = k * T;
  }
  __syncthreads();
  const int ready = own ? kend : s_flag[1];
  bool ok = true;
  auto issue = [&](int j) {
    const int k = k0 + j * TK;
    if (ok && k % T == 0 && k >= ready) {
      if (tid == 0) s_flag[0] = wait_ge(gate + k / T, 1, abort_flag) ? 1 : 0;
      __syncthreads();
      ok = s_flag[0] != 0;
    }
    if (ok)
      trtri_load<VEC>(As + (j % TST) * TA_SLAB, Bs + (j % TST) * TB_SLAB, Arow, rows, Bcol, cols, k, kend, ld, tid);
  };
#pragma unroll
  for (int st = 0; st < TST - 1; ++st) {
    if (st < nslab) issue(st);
    cp_async_commit();
  }
  for (int s = 0; s < nslab && ok; ++s) {
    cp_async_wait<TST - 2>();
    __syncthreads();
    const int nx = s + TST - 1;
    if (nx < nslab) issue(nx);
    cp_async_commit();
    const double* X = As + (s % TST) * TA_SLAB + sha;
    const double* Y = Bs + (s % TST) * TB_SLAB + shb;
#pragma unroll
    for (int kk = 0; kk < TK; kk += 4) {
      double a[2][2], bb[4];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi) {
        const int r = wm * 32 + mi * 16 + g;
        a[mi][0] = X[r * TSK + kk + t];
        a[mi][1] = X[(r + 8) * TSK + kk + t];
      }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) bb[ni] = Y[(kk + t) * TSN + wn * 32 + ni * 8 + g];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) dmma16x8x4(acc[mi][ni], a[mi][0], a[mi][1], bb[ni]);
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  return ok;
}

// Zeros above the diagonal tile of tile column c (wc columns).
__device__ __forceinline__ void zero_above(double* Oi, int b, int c, int wc, bool vec, int tid) {
  for (int idx = 2 * tid; idx < c * T * T; idx += 2 * THREADS) {
    double* z = Oi + (size_t)(idx >> 6) * b + c * T + (idx & 63);
    if (vec && (idx & 63) + 1 < wc) {
      *reinterpret_cast<double2*>(z) = make_double2(0.0, 0.0);
    } else {
      if ((idx & 63) < wc) z[0] = 0.0;
      if ((idx & 63) + 1 < wc) z[1] = 0.0;
    }
  }
}

// Inverses of lower-triangular blocks, tile by tile:
//   X(c, c) = Linv_cc,  X(p, c) = -Linv_pp sum_{k=c}^{p-1} L(p, k) X(k, c)   (p > c).
// The sums are bound by the FP64 tensor pipe.
// One task per tile, claimed by distance p - c from the diagonal (all blocks
// of all instances of a distance before the next one), so a task waits only
// on earlier tasks; it streams its sum as the tiles above it become final.  A
// task at distance 0 inverts the diagonal tile and clears its column above.
// Many blocks are done with a CTA per tile column instead, the longest first,
// after a launch for the diagonal tiles: no flags and no waits (tasks lose 7 %
// to them), but a serial chain of up to nq^2 / 2 tile products, which for few
// blocks outlasts everything else (16 blocks of 1117: 0.81 ms, by tiles 0.43).
// The columns are not claimed by resident CTAs: the SMs take a long, a middle
// and a short one each from the launch's order (claimed: 2 to 5 % slower).
template <bool COL>
__global__ void __launch_bounds__(THREADS, TRTRI_CTAS) block_trtri_kernel(const __grid_constant__ TrtriBatch B) {
  extern __shared__ __align__(16) double sm[];
  double* As = sm;
  double* Ys = sm + TRTRI_RING;
  __shared__ double rd[T];
  __shared__ int s_task[4], s_flag[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1, g = lane >> 2, t = lane & 3;
  int dist = COL ? 1 : 0, before = 0;  // thread 0: tasks of distances < dist
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      const int ti = COL ? (int)blockIdx.x : atomicAdd(B.counter, 1);
      s_task[0] = -1;
      while (ti < B.total) {
        const int len = B.nqmax - dist;  // COL: columns of len tiles below the diagonal one, the longest first
        int local = ti - before, cnt = 0, k = 0;
        for (; k < B.count; ++k) {
          const int nq = B.inst[k].nq;
          const int m = B.inst[k].n * (COL ? (nq > len ? 1 : 0) : max(0, nq - dist));
          if (local < m) break;
          local -= m;
          cnt += m;
        }
        if (k < B.count) {
          const int nq = B.inst[k].nq, w = COL ? 1 : nq - dist;
          s_task[0] = k;
          s_task[1] = local / w;
          s_task[2] = COL ? nq - 1 - len : local % w;
          s_task[3] = dist;
          break;
        }
        before += cnt;
        ++dist;
      }
    }
    __syncthreads();
    if (s_task[0] < 0) break;
    const TrtriDev& I = B.inst[s_task[0]];
    const int i = s_task[1], c = s_task[2];
    const int b = I.b, nq = I.nq;
    const double* Di = I.D + (size_t)i * b * b;
    double* Oi = I.out + (size_t)i * b * b;
    int* gate = B.flags + I.flag0 + ((size_t)i * nq + c) * nq;
    const int wc = min(T, b - c * T);
    // the task's (first) tile; its place is worked out here, where a task of one
    // tile takes 1 us less than with it inside the loop below
    const int p0 = COL ? c + 1 : c + s_task[3], rp0 = min(T, b - p0 * T);
    double* o0 = Oi + (size_t)(p0 * T) * b + c * T;
    const bool vec = ((b & 1) == 0) &&
                     (((reinterpret_cast<uintptr_t>(Di) | reinterpret_cast<uintptr_t>(Oi)) & 15) == 0);
    if (p0 == c) {  // never with COL
      if (vec) load_async<SG>(As, Di + (size_t)(c * T) * b + c * T, b, wc, wc, tid);
      else load<SG>(As, Di + (size_t)(c * T) * b + c * T, b, wc, wc, tid);
      cp_async_commit();
      if (!COL && B.zeros) zero_above(Oi, b, c, wc, vec, tid);
      cp_async_wait<0>();
      __syncthreads();
      for (int r = wc + tid; r < T; r += THREADS) As[r * SG + r] = 1.0;
      __syncthreads();
      trinv(As, Ys, rd, tid);
      for (int idx = tid; idx < T * T; idx += THREADS) {
        const int r = idx >> 6, cc = idx & 63;
        if (r < wc && cc < wc) o0[(size_t)r * b + cc] = Ys[r * SG + cc];
      }
      __syncthreads();
      if (tid == 0) st_release(gate + c, 1);
      continue;
    }
    // a tile, or the tiles of a column one after the other: those are read back
    // by this CTA alone (a barrier orders them)
    const bool own = COL && !B.zeros;  // COL: always
    const int pend = COL ? nq : p0 + 1;
    if (COL) zero_above(Oi, b, c, wc, vec, tid);
    for (int p = p0; p < pend; ++p) {
      const int rp = COL ? min(T, b - p * T) : rp0;
      double* o = COL ? Oi + (size_t)(p * T) * b + c * T : o0;
      double acc[2][4][4];
      zero_acc(acc);
      const double* Arow = Di + (size_t)(p * T) * b;
      // Linv_pp (a task of distance 0 wrote it) is fetched during the sum when
      // it is there already (for a column it always is)
      const double* Lpp = Oi + (size_t)(p * T) * b + p * T;
      const int* pgate = B.flags + I.flag0 + ((size_t)i * nq + p) * nq + p;
      if (!COL) {
        if (tid == 0) s_flag[0] = ld_acquire(pgate) >= 1;
        __syncthreads();
      }
      const bool fetched = COL || s_flag[0] != 0;
      auto fetch = [&]() {
        if (vec) load_async<SG>(Ys, Lpp, b, rp, rp, tid);
        else load_shifted_async<T, T, SG>(Ys, Lpp, b, rp, 0, rp, tid);
        cp_async_commit();
      };
      if (fetched) fetch();
      if (!(vec ? trtri_stream<true>(Arow, rp, Oi + c * T, wc, c * T, p * T, b, own, gate, B.abort_flag, s_flag, As,
                                          acc, tid, wm, wn, g, t)
                : trtri_stream<false>(Arow, rp, Oi + c * T, wc, c * T, p * T, b, own, gate, B.abort_flag, s_flag, As,
                                           acc, tid, wm, wn, g, t)))
        break;
      if (!fetched) {
        if (tid == 0) s_flag[0] = wait_ge(pgate, 1, B.abort_flag) ? 1 : 0;
        __syncthreads();
        if (!s_flag[0]) break;
        fetch();
      }
      // As[n][j] = acc[j][n] (the slab ring is free again)
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int j = wm * 32 + mi * 16 + g + h * 8;
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int e = 0; e < 2; ++e) As[(wn * 32 + ni * 8 + 2 * t + e) * SG + j] = acc[mi][ni][h * 2 + e];
        }
      cp_async_wait<0>();
      __syncthreads();
      // X = -Linv_pp acc: Linv_pp is lower triangular (row tile mi sums k < 16 (mi + 1));
      // a warp owns 16 whole columns, so the four have the same work
      const int shl = vec ? 0 : row_parity(Lpp, b, g);
      double x[4][2][4];
#pragma unroll
      for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 2; ++ni)
#pragma unroll
          for (int e = 0; e < 4; ++e) x[mi][ni][e] = 0.0;
#pragma unroll
      for (int kk = 0; kk < T; kk += 4) {
        const double b0 = As[(16 * warp + g) * SG + kk + t], b1 = As[(16 * warp + 8 + g) * SG + kk + t];
#pragma unroll
        for (int mi = kk / 16; mi < 4; ++mi) {
          const double* l = Ys + (16 * mi + g) * SG + kk + t + shl;
          const double a0 = l[0], a1 = l[8 * SG];
          dmma16x8x4(x[mi][0], a0, a1, b0);
          dmma16x8x4(x[mi][1], a0, a1, b1);
        }
      }
#pragma unroll
      for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = 16 * mi + g + h * 8;
          if (r >= rp) continue;
#pragma unroll
          for (int ni = 0; ni < 2; ++ni) {
            const int n = 16 * warp + ni * 8 + 2 * t;
            double* dst = o + (size_t)r * b + n;
            if (vec && n + 1 < wc) {
              *reinterpret_cast<double2*>(dst) = make_double2(-x[mi][ni][h * 2], -x[mi][ni][h * 2 + 1]);
            } else {
              if (n < wc) dst[0] = -x[mi][ni][h * 2];
              if (n + 1 < wc) dst[1] = -x[mi][ni][h * 2 + 1];
            }
          }
        }
      __syncthreads();
      if (!COL && tid == 0) st_release(gate + p, 1);
    }
    if (COL) break;
  }
}

__global__ void logdet_part_kernel(const double* D, int n, int b, const double* Tt, int a, double* part) {
  __shared__ double red[256];
  const int blk = blockIdx.x, tid = threadIdx.x;
  const double* M;
  int m;
  if (blk < n) {
    M = D + (size_t)blk * b * b;
    m = b;
  } else {
    M = Tt;
    m = a;
  }
  double s = 0.0;
  for (int k = tid; k < m; k += blockDim.x) s += log(M[(size_t)k * m + k]);
  red[tid] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (tid < o) red[tid] += red[tid + o];
    __syncthreads();
  }
  if (tid == 0) part[blk] = red[0];
}

__global__ void logdet_final_kernel(const double* part, int cnt, double* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < cnt; ++i) s += part[i];
    *out = 2.0 * s;
  }
}

}  // namespace

size_t block_trtri_flags(int n, int b) {
  const size_t nq = (size_t)(b + T - 1) / T;
  return (size_t)n * nq * nq + 4;
}

int block_trtri(const TrtriInst* inst, int count, int* flags, int* abort_flag, cudaStream_t s) {
  if (count < 1) return cudaSuccess;
  {
    const int e = ensure_smem_attr(reinterpret_cast<const void*>(block_trtri_kernel<false>), (int)TRTRI_SMEM);
    if (e != cudaSuccess) return e;
  }
  cudaError_t e = cudaSuccess;
  for (int k0 = 0; k0 < count; k0 += TRTRI_MAXI) {
    TrtriBatch B;
    std::memset(&B, 0, sizeof(B));
    long long total = 0, nflag = 0, diag = 0;
    double work = 0;  // tile products of the launch
    int nqmax = 0;
    for (int k = k0; k < std::min(count, k0 + TRTRI_MAXI); ++k) {
      TrtriDev& I = B.inst[B.count];
      I.D = inst[k].D;
      I.out = inst[k].out;
      I.n = inst[k].n;
      I.b = inst[k].b;
      I.nq = (I.b + T - 1) / T;
      I.flag0 = nflag;
      if (I.n <= 0 || I.b <= 0) continue;
      nflag += (long long)I.n * I.nq * I.nq;
      total += (long long)I.n * I.nq * (I.nq + 1) / 2;
      diag += (long long)I.n * I.nq;
      work += (double)I.n * I.nq * I.nq * I.nq / 6;
      nqmax = std::max(nqmax, I.nq);
      B.count++;
    }
    // Columns when every CTA slot has at least COLUMN_WORK times the tile
    // products of the longest column to do: tile by tile against column by
    // column, 12 x 20 blocks of 1500 (4.3 times) 10.78 and 10.05 ms, 100 of
    // 1500 (1.8) 4.55 and 4.18, 30 of 2500 (0.90) 5.95 and 5.62, 20 of 4000
    // (0.95) 14.6 and 14.0, 40 of 1500 (0.72) 1.88 and 1.85; 10 of 6000 (0.71)
    // 24.3 and 25.8, 14 of 4000 (0.66) 10.3 and 11.2, 20 of 1500 (0.36) 0.99 and
    // 1.52.  Blocks of one or two tiles gain nothing (1200 of 128: 0.124, 0.130).
    const int slots = TRTRI_CTAS * device_sm_count();
    const bool columns = nqmax > 2 && work >= COLUMN_WORK * (0.5 * nqmax * nqmax) * slots;
    if (total == 0) continue;
    if (total > INT32_MAX / 2) return cudaErrorInvalidValue;
    B.total = (int)(columns ? diag : total);
    B.zeros = columns ? 0 : 1;
    B.nqmax = nqmax;
    B.flags = flags;
    B.counter = flags + nflag;
    B.abort_flag = abort_flag;
    if ((e = cudaMemsetAsync(flags, 0, (nflag + 1) * sizeof(int), s)) != cudaSuccess) return e;
    {
      bta::ProfScope _ps(bta::PROF_TRTRI, s);
      block_trtri_kernel<false><<<std::min(B.total, slots), THREADS, TRTRI_SMEM, s>>>(B);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (!columns) continue;
    B.total = (int)diag;  // as many columns
    {
      const int rc = ensure_smem_attr(reinterpret_cast<const void*>(block_trtri_kernel<true>), (int)TRTRI_SMEM);
      if (rc != cudaSuccess) return rc;
    }
    {
      bta::ProfScope _ps(bta::PROF_TRTRI, s);
      block_trtri_kernel<true><<<B.total, THREADS, TRTRI_SMEM, s>>>(B);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

int logdet_launch(const double* D, int n, int b, const double* Tt, int a, double* part, double* out,
                  cudaStream_t s) {
  const int cnt = n + (a > 0 ? 1 : 0);
  if (cnt > 0) {
    bta::ProfScope _ps(bta::PROF_OTHER, s);
    logdet_part_kernel<<<cnt, 256, 0, s>>>(D, n, b, Tt, a, part);
  }
  {
    bta::ProfScope _ps(bta::PROF_OTHER, s);
    logdet_final_kernel<<<1, 32, 0, s>>>(part, cnt, out);
  }
  return cudaGetLastError();
}

}  // namespace bta
