// Matrix algebra of the LNV chain on device-resident block matrices:
//   matrix_scale / matrix_sum (same range: scal + axpy, src/mult_module.f90:2677-2738)
//   matrix_add / addscan       (different ranges, src/multiply_module.f90:807-943):
//                               a = alpha*a + beta*b on the blocks both ranges store
//   matrix_transpose           (src/mult_module.f90:2609-2673 via the retro/transposed addresses)
//   matrix_trace / matrix_product_trace (src/mult_module.f90:2773-2916)
//   GetHLimits                 (src/McWeeny.f90:1020-1109)
// Elementwise kernels are HBM-bound grid-stride loops with 16-byte accesses;
// the reductions are two-level with a fixed grid, so results are identical
// from run to run.
#include <climits>
#include <functional>
#include <cmath>
#include <limits>

#include "cq_internal.hpp"

namespace cqb {
namespace {

constexpr int kT = 256;
constexpr int kRedBlocks = 592;    // 148 SMs x 4: the largest grid of one exact sum

int grid_for(int64_t n) {
  int64_t b = (n + kT - 1) / kT;
  return (int)std::min<int64_t>(std::max<int64_t>(b, 1), 148 * 16);
}

__global__ void k_scale(double* __restrict__ a, int64_t n, double alpha) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] = __dmul_rn(a[i], alpha);
}
// a = a + fl(beta*b)  (daxpy with separate rounding of the product)
__global__ void k_axpy(double* __restrict__ a, int64_t n, double beta, const double* __restrict__ b) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] = __dadd_rn(a[i], __dmul_rn(beta, b[i]));
}
// a = fl(fl(alpha*a) + fl(beta*b)): k_scale followed by k_axpy in one pass (same roundings);
// 16-byte accesses when both arrays are 16-byte aligned
__global__ void k_axpby(double* __restrict__ a, int64_t n, double alpha, double beta, const double* __restrict__ b,
                        int vec) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (vec) {
    double2* a2 = reinterpret_cast<double2*>(a);
    const double2* b2 = reinterpret_cast<const double2*>(b);
    for (int64_t i = i0; i < n / 2; i += stride) {
      double2 x = a2[i], y = b2[i];
      x.x = __dadd_rn(__dmul_rn(x.x, alpha), __dmul_rn(beta, y.x));
      x.y = __dadd_rn(__dmul_rn(x.y, alpha), __dmul_rn(beta, y.y));
      a2[i] = x;
    }
    if (i0 == 0 && (n & 1)) a[n - 1] = __dadd_rn(__dmul_rn(a[n - 1], alpha), __dmul_rn(beta, b[n - 1]));
  } else {
    for (int64_t i = i0; i < n; i += stride) a[i] = __dadd_rn(__dmul_rn(a[i], alpha), __dmul_rn(beta, b[i]));
  }
}
// matched blocks: a = fl(alpha*a) + fl(beta*b); unmatched blocks of a are left as they are
__global__ void k_masked_add(int nnz, const int* __restrict__ partner, const int64_t* __restrict__ a_elem,
                             const int64_t* __restrict__ b_elem, const int* __restrict__ row, const int* __restrict__ cover,
                             const int* __restrict__ prim_nsf, const int* __restrict__ cover_nsf, double* __restrict__ a,
                             double alpha, const double* __restrict__ b, double beta) {
  int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (e >= nnz) return;
  int pb = partner[e];
  if (pb < 0) return;
  int ne = prim_nsf[row[e]] * cover_nsf[cover[e]];
  double* A = a + a_elem[e];
  const double* B = b + b_elem[pb];
  for (int t = lane; t < ne; t += 32) A[t] = __dadd_rn(__dmul_rn(alpha, A[t]), __dmul_rn(beta, B[t]));
}
// the same for uniform 4 x 4 blocks with 16-byte aligned arrays: eight lanes per block, one double2 each (a warp per
// block would leave half of its lanes idle and look up four index arrays per block)
__global__ void __launch_bounds__(kT) k_masked_add_nd4(int nnz, const int* __restrict__ partner, double2* __restrict__ a,
                                                       double alpha, const double2* __restrict__ b, double beta) {
  const int64_t stride = (int64_t)gridDim.x * kT;
  for (int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x; i < (int64_t)nnz * 8; i += stride) {
    const int pb = partner[i >> 3];
    if (pb < 0) continue;
    double2 x = a[i];
    const double2 y = b[(int64_t)pb * 8 + (i & 7)];
    x.x = __dadd_rn(__dmul_rn(alpha, x.x), __dmul_rn(beta, y.x));
    x.y = __dadd_rn(__dmul_rn(alpha, x.y), __dmul_rn(beta, y.y));
    a[i] = x;
  }
}
// AT(dest) = A(e)^T: a warp per block.  STAGED: through shared memory, so that both the read and the write run along
// memory; else each lane writes its elements where they belong, one round trip less (see dev_transpose).
template <bool STAGED>
__global__ void __launch_bounds__(kT) k_transpose(int nnz, const int* __restrict__ dest, const int64_t* __restrict__ elem,
                                                  const int* __restrict__ row, const int* __restrict__ cover,
                                                  const int* __restrict__ prim_nsf, const int* __restrict__ cover_nsf,
                                                  const double* __restrict__ a, double* __restrict__ at) {
  int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (e >= nnz) return;
  const int ndi = prim_nsf[row[e]], ndj = cover_nsf[cover[e]], ne = ndi * ndj;
  const double* A = a + elem[e];
  double* T = at + elem[dest[e]];
  if constexpr (STAGED) {
    __shared__ double tile[kT / 32][16 * 17];
    double* W = tile[threadIdx.x >> 5];
    const int pad = ~ndi & 1, ld = ndi + pad;              // odd column distance: the reads along a row hit different banks
    const int by_j = 65536 / ndj + 1;                      // t / ndj = t * by_j >> 16 for t < 256, ndj <= 16
    if (pad) {
      const int by_i = 65536 / ndi + 1;
      for (int t = lane; t < ne; t += 32) W[t + ((t * by_i) >> 16)] = A[t];
    } else {
      for (int t = lane; t < ne; t += 32) W[t] = A[t];
    }
    __syncwarp();
    for (int t = lane; t < ne; t += 32) {                  // element (n2, n1) of the transpose
      const int n1 = (t * by_j) >> 16, n2 = t - n1 * ndj;
      T[t] = W[n1 + ld * n2];
    }
  } else {
    for (int t = lane; t < ne; t += 32) {
      const int n1 = t % ndi, n2 = t / ndi;
      T[n2 + ndj * n1] = A[t];
    }
  }
}
// the same for uniform 4 x 4 blocks with 16-byte aligned arrays: eight lanes per block; lane (n1 pair, n2) reads two
// values of column n2 and trades one with the lane of column n2 ^ 1, so that it writes two neighbours as well.
// Memory bound: 151 MB read and written (42-bohr range of 512 atoms) in 54.9 us against 236.9 us with a warp per block.
__global__ void __launch_bounds__(kT) k_transpose_nd4(int nnz, const int* __restrict__ dest, const double2* __restrict__ a,
                                                      double2* __restrict__ at) {
  const int64_t stride = (int64_t)gridDim.x * kT, n = (int64_t)nnz * 8;
  const int64_t n32 = (n + 31) & ~(int64_t)31;            // whole warps: the shuffle needs every lane
  for (int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x; i < n32; i += stride) {
    const double2 v = i < n ? a[i] : make_double2(0.0, 0.0);
    const int r = (int)(i & 1), c = (int)(i >> 1) & 3;     // rows 2r, 2r + 1 of column c
    const double got = __shfl_xor_sync(0xffffffffu, c & 1 ? v.x : v.y, 2);
    // even column: row 2r of columns c, c + 1; odd column: row 2r + 1 of columns c - 1, c
    const double2 w = c & 1 ? make_double2(got, v.y) : make_double2(v.x, got);
    if (i < n) at[(int64_t)dest[i >> 3] * 8 + 2 * (2 * r + (c & 1)) + (c >> 1)] = w;
  }
}
// ---------------------------------------------------------------------------
// Exact, order-independent sums (matrix_product_trace / matrix_trace).
// Every term (a rounded product x*y, or an element) is converted exactly to a
// 192-bit two's-complement fixed-point integer whose least significant bit is
// 2^(emax-150), emax being the largest binary exponent among the terms (pass 1).
// Integer addition is associative, so the sum does not depend on the grid or on
// the order of the terms; the host rounds it once to the nearest double.
// Terms below 2^(emax-150) are truncated toward zero (relative effect < n 2^-150).
// ---------------------------------------------------------------------------
constexpr int kAccFrac = 150;   // fraction bits kept below the largest term's exponent
constexpr int kSumSlots = 32;   // exact sums fetched together by dev_dots
constexpr int kEBias = 2048;    // exponent bias of the pass-1 maximum (frexp exponents lie in [-1073, 1024])

struct Acc192 { uint64_t w[3]; };

__device__ __forceinline__ void acc_add(Acc192& a, const Acc192& b) {
  uint64_t s0 = a.w[0] + b.w[0];
  uint64_t c0 = s0 < a.w[0];
  uint64_t s1 = a.w[1] + b.w[1];
  uint64_t c1 = s1 < a.w[1];
  uint64_t s1c = s1 + c0;
  c1 += s1c < s1;
  a.w[0] = s0; a.w[1] = s1c; a.w[2] = a.w[2] + b.w[2] + c1;
}
// term v -> fixed point with lsb 2^lsb_exp (exact for every bit at or above the lsb)
__device__ __forceinline__ void acc_term(Acc192& a, double v, int lsb_exp) {
  const uint64_t u = (uint64_t)__double_as_longlong(v);
  const int ef = (int)(u >> 52) & 0x7ff;
  uint64_t mag = u & 0xfffffffffffffull;                // v = mag 2^(max(ef, 1) - 1075)
  if (ef) mag |= 1ull << 52;
  if (mag == 0) return;
  const int s = (ef ? ef : 1) - 1075 - lsb_exp;         // bit position of mag's lsb
  Acc192 t = {{0, 0, 0}};
  if (s >= 0) {
    const int idx = s >> 6, off = s & 63;
    const uint64_t lo = mag << off, hi = off ? mag >> (64 - off) : 0;
    t.w[0] = idx == 0 ? lo : 0;
    t.w[1] = idx == 1 ? lo : idx == 0 ? hi : 0;
    t.w[2] = idx == 2 ? lo : idx == 1 ? hi : 0;
  } else if (-s < 64) {
    t.w[0] = mag >> (-s);
  }
  if (u >> 63) {                                        // two's complement negation
    t.w[0] = ~t.w[0]; t.w[1] = ~t.w[1]; t.w[2] = ~t.w[2];
    Acc192 one = {{1, 0, 0}};
    acc_add(t, one);
  }
  acc_add(a, t);
}
__device__ __forceinline__ double dterm(const double* x, const double* y, int64_t i) {
  return y ? __dmul_rn(x[i], y[i]) : x[i];
}
// The sums of one call: operands, lengths and grid of each.
struct SumArgs {
  const double* x[kSumSlots];
  const double* y[kSumSlots];
  int64_t n[kSumSlots];
  int blocks[kSumSlots];
};
// Scratch of a sum: flags (largest biased exponent, non-finite, blocks done), zero between calls (the last block of
// pass 2 clears them), and the block partials.
constexpr int kSumFlags = 3;

// pass 1 of sum blockIdx.y: largest frexp exponent of the nonzero terms, stored biased by kEBias (0 = every term is
// zero); a non-finite term sets the flag
__global__ void __launch_bounds__(kT) k_acc_emax(const __grid_constant__ SumArgs A, int* __restrict__ flags) {
  const int k = blockIdx.y;
  if (blockIdx.x >= A.blocks[k]) return;
  const double *x = A.x[k], *y = A.y[k];
  const int64_t n = A.n[k], stride = (int64_t)A.blocks[k] * kT;
  int best = 0;
  bool bad = false;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x; i < n; i += stride) {
    const uint64_t u = (uint64_t)__double_as_longlong(dterm(x, y, i));
    const int ef = (int)(u >> 52) & 0x7ff;
    const uint64_t frac = u & 0xfffffffffffffull;
    if (ef == 0x7ff) bad = true;
    else if (ef) best = max(best, ef - 1022 + kEBias);
    else if (frac) best = max(best, 64 - __clzll((long long)frac) - 1074 + kEBias);
  }
  best = __reduce_max_sync(0xffffffffu, best);
  if ((threadIdx.x & 31) == 0 && best != 0) atomicMax(flags + kSumFlags * k, best);
  if (bad) atomicExch(flags + kSumFlags * k + 1, 1);
}
// sum over the block of every thread's a, valid in thread 0
__device__ Acc192 block_acc_reduce(Acc192 a) {
  __shared__ uint64_t s[3][kT / 32];
  for (int o = 16; o; o >>= 1) {
    Acc192 z;
    for (int k = 0; k < 3; ++k) z.w[k] = __shfl_down_sync(0xffffffffu, a.w[k], o);
    acc_add(a, z);
  }
  const int warp = threadIdx.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) for (int k = 0; k < 3; ++k) s[k][warp] = a.w[k];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kT / 32; ++w) {
      const Acc192 z = {{s[0][w], s[1][w], s[2][w]}};
      acc_add(a, z);
    }
  return a;
}
// pass 2 of sum blockIdx.y: fixed-point accumulation, one 192-bit partial per block (zero when pass 1 found no
// nonzero term or a non-finite one: the host reports 0 or NaN from the flags); the block that finishes last adds the
// partials into out[4 k .. 4 k + 2], puts the flags into out[4 k + 3] and clears them.  What bounds the two passes for
// the chain's matrices is launches and their gaps: all sums of a call share the two launches, and `out` is pinned
// host memory, so no memset, final pass or copy follows them.
__global__ void __launch_bounds__(kT) k_acc_sum(const __grid_constant__ SumArgs A, int* __restrict__ flags,
                                                uint64_t* __restrict__ part, int part_stride, uint64_t* __restrict__ out) {
  __shared__ int last;
  const int k = blockIdx.y, nb = A.blocks[k];
  if (blockIdx.x >= nb) return;
  const double *x = A.x[k], *y = A.y[k];
  const int64_t n = A.n[k], stride = (int64_t)nb * kT;
  int* f = flags + kSumFlags * k;
  uint64_t* p = part + (size_t)k * part_stride;
  const int eb = f[0], bad = f[1];
  Acc192 a = {{0, 0, 0}};
  if (eb != 0 && bad == 0) {
    const int lsb = eb - kEBias - kAccFrac;
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x; i < n; i += stride) acc_term(a, dterm(x, y, i), lsb);
  }
  a = block_acc_reduce(a);
  if (threadIdx.x == 0) {
    for (int w = 0; w < 3; ++w) p[3 * blockIdx.x + w] = a.w[w];
    __threadfence();
    last = atomicAdd(f + 2, 1) == nb - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  Acc192 t = {{0, 0, 0}};
  for (int b = threadIdx.x; b < nb; b += kT) {
    const Acc192 z = {{__ldcg(p + 3 * b), __ldcg(p + 3 * b + 1), __ldcg(p + 3 * b + 2)}};
    acc_add(t, z);
  }
  t = block_acc_reduce(t);
  if (threadIdx.x == 0) {
    for (int w = 0; w < 3; ++w) out[4 * k + w] = t.w[w];
    out[4 * k + 3] = (uint64_t)(uint32_t)eb | ((uint64_t)(uint32_t)bad << 32);
    f[0] = f[1] = f[2] = 0;
  }
}
// store_matrix_value(..., j, j, one) on every onsite block: the diagonal of each atom's self block
__global__ void k_set_onsite_diag(int n_prim, const int64_t* __restrict__ onsite, const int* __restrict__ prim_nsf,
                                  double value, double* __restrict__ a) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_prim) return;
  const int nd = prim_nsf[p];
  for (int j = 0; j < nd; ++j) a[onsite[p] + j * nd + j] = value;
}
// onsite diagonal elements gathered for the exact trace
__global__ void k_gather_diag(int n_prim, const int64_t* __restrict__ onsite, const int* __restrict__ prim_nsf,
                              const int* __restrict__ diag_off, const double* __restrict__ a, double* __restrict__ out) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_prim) return;
  int nd = prim_nsf[p];
  for (int j = 0; j < nd; ++j) out[diag_off[p] + j] = a[onsite[p] + j * nd + j];
}
// GetHLimits: per primary atom and column orbital i, HMin_i = sum(+-|H|), HMax_i = sum |H|
// (onsite block adds |H| to both); min/max over atoms are order independent.
__global__ void k_hlimits(int n_prim, const int* __restrict__ row_ptr, const int64_t* __restrict__ nb_elem,
                          const int* __restrict__ nb_cover, const int64_t* __restrict__ onsite,
                          const int* __restrict__ prim_nsf, const int* __restrict__ cover_nsf, const double* __restrict__ h,
                          double* __restrict__ hmin_atom, double* __restrict__ hmax_atom) {
  int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (p >= n_prim) return;
  const int nsfi = prim_nsf[p];
  double mn = 0.0, mx = 0.0;
  for (int e = row_ptr[p]; e < row_ptr[p + 1]; ++e) {
    int nsfj = cover_nsf[nb_cover[e]];
    const double* H = h + nb_elem[e];
    bool on = nb_elem[e] == onsite[p];
    if (lane < nsfj) {
      for (int j = 0; j < nsfi; ++j) {
        double v = fabs(H[j + nsfi * lane]);
        mn = on ? mn + v : mn - v;
        mx = mx + v;
      }
    }
  }
  double amn = 1.0e30, amx = -1.0e30;
  if (lane < nsfi) { amn = mn; amx = mx; }
  for (int o = 16; o; o >>= 1) {
    amn = fmin(amn, __shfl_down_sync(0xffffffffu, amn, o));
    amx = fmax(amx, __shfl_down_sync(0xffffffffu, amx, o));
  }
  if (lane == 0) { hmin_atom[p] = amn; hmax_atom[p] = amx; }
}
__global__ void k_minmax(const double* __restrict__ mn, const double* __restrict__ mx, int n, double* __restrict__ out) {
  __shared__ double smn[kT], smx[kT];
  double a = 1.0e30, b = -1.0e30;
  for (int i = threadIdx.x; i < n; i += kT) { a = fmin(a, mn[i]); b = fmax(b, mx[i]); }
  smn[threadIdx.x] = a; smx[threadIdx.x] = b;
  __syncthreads();
  for (int w = kT / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) { smn[threadIdx.x] = fmin(smn[threadIdx.x], smn[threadIdx.x + w]); smx[threadIdx.x] = fmax(smx[threadIdx.x], smx[threadIdx.x + w]); }
    __syncthreads();
  }
  if (threadIdx.x == 0) { out[0] = smn[0]; out[1] = smx[0]; }
}

}  // namespace

void dev_scale(System& S, double* a, int64_t n, double alpha) {
  if (n <= 0) return;
  k_scale<<<grid_for(n), kT, 0, S.stream>>>(a, n, alpha);
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}
void dev_axpy(System& S, double* a, int64_t n, double beta, const double* b) {
  if (n <= 0) return;
  k_axpy<<<grid_for(n), kT, 0, S.stream>>>(a, n, beta, b);
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}
void dev_axpby(System& S, double* a, int64_t n, double alpha, double beta, const double* b) {
  if (n <= 0) return;
  const int vec = ((uintptr_t)a % 16 == 0) && ((uintptr_t)b % 16 == 0);
  k_axpby<<<grid_for(vec ? (n + 1) / 2 : n), kT, 0, S.stream>>>(a, n, alpha, beta, b, vec);
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}
void dev_copy(System& S, double* dst, const double* src, int64_t n) {
  if (n <= 0 || dst == src) return;
  CQ_CUDA(cudaMemcpyAsync(dst, src, sizeof(double) * n, cudaMemcpyDeviceToDevice, S.stream));
}
void dev_matrix_add(System& S, int ra, double* a, double alpha, int rb, const double* b, double beta) {
  RangeIndex &A = *S.ranges[ra], &B = *S.ranges[rb];
  AddMap& m = get_addmap(S, ra, rb);
  if (A.nnz == 0) return;
  if (S.uniform_nsf == 4 && ((uintptr_t)a | (uintptr_t)b) % 16 == 0)
    k_masked_add_nd4<<<grid_for((int64_t)A.nnz * 8), kT, 0, S.stream>>>(
        A.nnz, m.partner.p, reinterpret_cast<double2*>(a), alpha, reinterpret_cast<const double2*>(b), beta);
  else
    k_masked_add<<<(int)(((int64_t)A.nnz * 32 + kT - 1) / kT), kT, 0, S.stream>>>(
        A.nnz, m.partner.p, A.nb_elem.p, B.nb_elem.p, A.nb_row.p, A.nb_cover.p, S.dg.prim_nsf.p, S.dg.cover_nsf.p, a, alpha,
        b, beta);
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}
void dev_transpose(System& S, int r, const double* a, double* at) {
  RangeIndex& R = *S.ranges[r];
  CQ_CHECK(a != at, CQ_ERR_ARG, "transpose cannot run in place");
  if (R.nnz == 0) return;
  if (S.uniform_nsf == 4 && ((uintptr_t)a | (uintptr_t)at) % 16 == 0)
    k_transpose_nd4<<<grid_for((int64_t)R.nnz * 8), kT, 0, S.stream>>>(
        R.nnz, R.trans_dest.p, reinterpret_cast<const double2*>(a), reinterpret_cast<double2*>(at));
  else {
    // staged from a mean of 110 elements per block on (512 atoms, 16-bohr range, staged / direct, us): 13 x 13 36.4 / 45.0,
    // 16 x 16 44.6 / 74.7 (79.0 before its columns were padded in shared memory), 11 x 11 34.7 / 35.6, 10 x 10 31.3 / 24.9,
    // 4 and 13 rows 14.7 / 12.5, 1 and 4 rows 12.1 / 8.9
    auto* kern = R.length >= (int64_t)110 * R.nnz ? k_transpose<true> : k_transpose<false>;
    kern<<<(int)(((int64_t)R.nnz * 32 + kT - 1) / kT), kT, 0, S.stream>>>(
        R.nnz, R.trans_dest.p, R.nb_elem.p, R.nb_row.p, R.nb_cover.p, S.dg.prim_nsf.p, S.dg.cover_nsf.p, a, at);
  }
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}
// Round a 192-bit two's-complement fixed-point value (lsb = 2^lsb_exp) to the nearest double, ties to even.
double acc192_to_double(const uint64_t in[3], int lsb_exp) {
  uint64_t w[3] = {in[0], in[1], in[2]};
  bool neg = (w[2] >> 63) != 0;
  if (neg) {
    w[0] = ~w[0]; w[1] = ~w[1]; w[2] = ~w[2];
    if (++w[0] == 0 && ++w[1] == 0) ++w[2];
  }
  int h = -1;
  for (int k = 2; k >= 0 && h < 0; --k)
    if (w[k]) h = 64 * k + 63 - __builtin_clzll(w[k]);
  if (h < 0) return 0.0;
  auto bit = [&](int b) -> uint64_t { return b < 0 ? 0 : (w[b >> 6] >> (b & 63)) & 1u; };
  uint64_t m = 0;
  int sh = h > 52 ? h - 52 : 0;                  // bits dropped below the 53-bit mantissa
  for (int b = h; b >= sh; --b) m = (m << 1) | bit(b);
  if (sh > 0) {
    uint64_t half = bit(sh - 1), sticky = 0;
    for (int b = sh - 2; b >= 0 && !sticky; --b) sticky |= bit(b);
    if (half && (sticky || (m & 1))) ++m;         // may carry to 2^53, still exact in a double
  }
  double v = std::ldexp((double)m, lsb_exp + sh);
  return neg ? -v : v;
}

// Grid of an exact sum: integer accumulation is associative, so the grid only sets the
// parallelism (about four elements per thread, at most 148 SMs x 4 blocks).
static int acc_grid(int64_t n) {
  int64_t g = (n + 4 * kT - 1) / (4 * kT);
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, kRedBlocks));
}

// Enqueue the two passes of up to kSumSlots sums; the 4-word results (3 fixed-point words, flags) land in res.
static void exact_sums_launch(int count, const double* const* x, const double* const* y, const int64_t* n, int* flags,
                              uint64_t* part, uint64_t* res, cudaStream_t st) {
  SumArgs A;
  int grid = 1;
  for (int k = 0; k < count; ++k) {
    A.x[k] = x[k]; A.y[k] = y ? y[k] : nullptr; A.n[k] = n[k]; A.blocks[k] = acc_grid(n[k]);
    grid = std::max(grid, A.blocks[k]);
  }
  k_acc_emax<<<dim3(grid, count), kT, 0, st>>>(A, flags);
  k_acc_sum<<<dim3(grid, count), kT, 0, st>>>(A, flags, part, 3 * kRedBlocks, res);
  CQ_CUDA(cudaGetLastError());
}

// Value of a 4-word exact-sum result (k_acc_sum layout).
static double exact_sum_value(const uint64_t r[4]) {
  const int eb = (int)(uint32_t)(r[3] & 0xffffffffu);
  if ((r[3] >> 32) != 0) return std::numeric_limits<double>::quiet_NaN();
  if (eb == 0) return 0.0;
  return acc192_to_double(r, eb - kEBias - kAccFrac);
}

// Scratch of the exact sums: the block partials of every sum of a call (kept: the calls of a system follow one
// another on its stream) and the flags, zero between calls.
static void acc_scratch(System& S) {
  if (S.acc_part.n == 0) {
    S.acc_part.alloc((size_t)3 * kRedBlocks * kSumSlots, S.stream);
    S.acc_flags.alloc(kSumFlags * kSumSlots, S.stream);
    CQ_CUDA(cudaMemsetAsync(S.acc_flags.p, 0, sizeof(int) * kSumFlags * kSumSlots, S.stream));
  }
  if (!S.host_res) S.host_res = pinned_get();
}

void dev_dots_enqueue(System& S, int count, const double* const* x, const double* const* y, const int64_t* n) {
  CQ_CHECK(count >= 0 && count <= kSumSlots, CQ_ERR_ARG, "too many sums in one batch");
  if (count == 0) return;
  acc_scratch(S);
  static_assert(4 * kSumSlots <= kPinnedWords, "pinned result buffer too small");
  exact_sums_launch(count, x, y, n, S.acc_flags.p, S.acc_part.p, S.host_res, S.stream);
  S.launches += 2;
}

void dev_dots_fetch(System& S, int count, double* out) {
  if (count == 0) return;
  host_wait(S);
  for (int k = 0; k < count; ++k) out[k] = exact_sum_value(&S.host_res[4 * k]);
}

void dev_dots(System& S, int count, const double* const* x, const double* const* y, const int64_t* n, double* out) {
  dev_dots_enqueue(S, count, x, y, n);
  dev_dots_fetch(S, count, out);
}

double dev_dot(System& S, const double* x, const double* y, int64_t n) {
  double v = 0.0;
  dev_dots(S, 1, &x, &y, &n, &v);
  return v;
}

double dev_trace(System& S, int r, const double* a) {
  RangeIndex& R = *S.ranges[r];
  const int N = S.geo.n_prim;
  if (S.diag_off.n == 0) {
    std::vector<int> off(N + 1, 0);
    for (int p = 0; p < N; ++p) off[p + 1] = off[p] + S.geo.nsf[S.geo.prim_global[p]];
    S.diag_off.upload(off, S.stream);
    S.diag_buf.alloc(std::max(off[N], 1), S.stream);
  }
  k_gather_diag<<<(N + kT - 1) / kT, kT, 0, S.stream>>>(N, R.onsite.p, S.dg.prim_nsf.p, S.diag_off.p, a, S.diag_buf.p);
  S.launches++;
  CQ_CUDA(cudaGetLastError());
  return dev_dot(S, S.diag_buf.p, nullptr, (int64_t)S.diag_buf.n);
}
void dev_set_onsite_diag(System& S, int r, double* a, double value) {
  RangeIndex& R = *S.ranges[r];
  const int N = S.geo.n_prim;
  if (N == 0) return;
  k_set_onsite_diag<<<(N + kT - 1) / kT, kT, 0, S.stream>>>(N, R.onsite.p, S.dg.prim_nsf.p, value, a);
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}
void dev_h_limits(System& S, int r, const double* h, double* hmin, double* hmax) {
  RangeIndex& R = *S.ranges[r];
  int N = S.geo.n_prim;
  DevBuf<double> mn, mx, out;
  mn.alloc(N, S.stream); mx.alloc(N, S.stream); out.alloc(2, S.stream);
  k_hlimits<<<(N * 32 + kT - 1) / kT, kT, 0, S.stream>>>(N, R.row_ptr.p, R.nb_elem.p, R.nb_cover.p, R.onsite.p,
                                                       S.dg.prim_nsf.p, S.dg.cover_nsf.p, h, mn.p, mx.p);
  k_minmax<<<1, kT, 0, S.stream>>>(mn.p, mx.p, N, out.p);
  S.launches += 2;
  CQ_CUDA(cudaGetLastError());
  double o[2];
  CQ_CUDA(cudaMemcpyAsync(o, out.p, sizeof(o), cudaMemcpyDeviceToHost, S.stream));
  host_wait(S);
  *hmin = o[0];
  *hmax = o[1];
}

// ---------------------------------------------------------------------------
// Exact dot products without any device allocation (cq_exact_dots_noalloc).
//
// Some callers cannot allocate device memory at the moment they need a trace: a Fortran/MPI
// host that has given the whole device to its own memory pool, or a latency-critical loop that
// must not take the device-wide synchronisation cudaMalloc and cudaFree can imply.  This entry
// point runs the same two kernels as the library's traces, with their scratch (block
// partials, results and flags) in one static device array instead of library-allocated memory.
// Every call uses that same array, so calls that overlap on the GPU (from two streams or two
// threads) race on it.
// ---------------------------------------------------------------------------
namespace {
constexpr int kNoAllocSums = CQ_NOALLOC_MAX_SUMS;
// words: block partials of two sums | 4-word result per sum | 3 int flags per sum
constexpr int kNoAllocPairs = 2;                                   // sums whose passes share two launches
constexpr int kNoAllocFlags = (kSumFlags * kNoAllocSums + 1) / 2;   // words
constexpr int kNoAllocWords = 3 * kRedBlocks * kNoAllocPairs + 4 * kNoAllocSums + kNoAllocFlags;
static __device__ __align__(256) uint64_t g_noalloc_scratch[kNoAllocWords];   // 28.1 KiB per device

// Device address of the static scratch on the current device.  The host-side name of the array
// is not a device address, so it is looked up with cudaGetSymbolAddress on every call (cheap, and
// it allocates nothing): a cached address would go stale if the host tore the context down
// (cudaDeviceReset) between calls.
uint64_t* noalloc_scratch() {
  void* p = nullptr;
  CQ_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
  return static_cast<uint64_t*>(p);
}
}  // namespace

int guarded_call(const std::function<void()>& f);   // capi.cpp: exceptions to status codes

}  // namespace cqb

extern "C" int cq_exact_dots_noalloc(int count, const double* const* x_dev, const double* const* y_dev,
                                     const int64_t* n, void* stream, double* out) {
  using namespace cqb;
  return guarded_call([&] {
    CQ_CHECK(x_dev && n && out, CQ_ERR_ARG, "null argument");
    CQ_CHECK(count >= 1 && count <= kNoAllocSums, CQ_ERR_ARG,
             "cq_exact_dots_noalloc: count must be 1..CQ_NOALLOC_MAX_SUMS (8) sums per call");
    for (int k = 0; k < count; ++k) CQ_CHECK(n[k] >= 0 && (x_dev[k] || n[k] == 0), CQ_ERR_ARG, "bad operand");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint64_t* base = noalloc_scratch();
    uint64_t* part = base;
    uint64_t* res = base + 3 * kRedBlocks * kNoAllocPairs;
    int* flags = reinterpret_cast<int*>(res + 4 * kNoAllocSums);
    // the flags (largest exponent, non-finite, blocks done) start at zero; the partials and results
    // are overwritten by every call
    CQ_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * kSumFlags * count, st));
    for (int k = 0; k < count; k += kNoAllocPairs)
      exact_sums_launch(std::min(kNoAllocPairs, count - k), x_dev + k, y_dev ? y_dev + k : nullptr, n + k,
                        flags + kSumFlags * k, part, res + 4 * k, st);
    uint64_t w[4 * kNoAllocSums];
    CQ_CUDA(cudaMemcpyAsync(w, res, sizeof(uint64_t) * 4 * count, cudaMemcpyDeviceToHost, st));
    CQ_CUDA(cudaStreamSynchronize(st));
    for (int k = 0; k < count; ++k) out[k] = exact_sum_value(&w[4 * k]);
  });
}

