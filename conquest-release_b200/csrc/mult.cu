// FP64 block-sparse products on the pair lists built in index.cu.
//
// Output stationary: each output block is owned by one group of lanes (one
// lane per element) that walks the block's (operand, B) pair list in the
// reference's order, so every element sees exactly the operation sequence of
// the default kernel (src/multiply_kernel_default.f90:204-214 for type 1,
// 390-402 for type 2):
//   type 1  c(n1,n2) = sum over k (A-halo order) of sum_n3 a(n1,n3) * b(n3,n2)
//   type 2  a(n1,n3) = sum over j (B-neighbour order) of sum_n2 c(n1,n2) * b(n3,n2)
// With `exact` the multiply and the add of every term round separately, which
// reproduces the default kernel built without FMA contraction bit for bit.
// No atomics, no reduction trees: results are deterministic and independent of
// the launch shape.
//
// The bound is the L2/HBM traffic of the operand blocks (an nd x nd FP64 block
// pair per triple, 2 nd^3 flops): for nd = 4 this is 256 B per 128 flops.  The 4 x 4 kernels write
// their output blocks with streaming (evict-first) stores, and every kernel reads its pair list (8
// bytes per triple, each read once) with streaming loads: an output range and a pair list are often
// larger than L2 (the 42-bohr range of the 512-atom cell: 152 MB; the pair list of LS.L -> LSL: 272 MB)
// and would otherwise push the operand blocks, which every output block re-reads, out of L2.
#include <algorithm>
#include <memory>

#include "cq_internal.hpp"

namespace cqb {
namespace {

template <bool EXACT>
__device__ __forceinline__ double madd(double acc, double x, double y) {
  if (EXACT) return __dadd_rn(acc, __dmul_rn(x, y));
  return fma(x, y, acc);
}

struct MultArgs {
  const int64_t* __restrict__ ptr;   // [n_out+1]
  const int2* __restrict__ pairs;    // (x block, b block)
  int n_out;
  // output blocks
  const int* __restrict__ o_row;
  const int* __restrict__ o_cover;
  const int64_t* __restrict__ o_elem;
  // first operand blocks (type 1: A; type 2: the input c)
  const int* __restrict__ x_cover;
  const int64_t* __restrict__ x_elem;
  // B blocks
  const int64_t* __restrict__ b_elem;
  const int* __restrict__ b_cover;
  const int* __restrict__ prim_nsf;
  const int* __restrict__ cover_nsf;
  const double* __restrict__ x;
  const double* __restrict__ b;
  double* __restrict__ out;
};

// Any block sizes (nd <= 16): one warp per output block, R elements per lane (32 R >= the largest block), operands read
// from global memory.  What bounds it: the chain of dependent loads of a pair (pair list, block offsets, inner dimension,
// values), so the next pair's offsets are looked up while the current one's values are on their way, and the list is read
// a pair further ahead.  It is the kernel of small blocks in products with few output blocks, where the group kernel
// waits for its staging (see auto_variant).  u: the block size when the whole system has one, else 0.
// Measured (6298 output blocks, type 2, 47 terms each; us): 5 x 5 blocks 50.3, without the look-ahead 99.5 and 113.2
// for the group kernel; blocks of 1 and 4 rows 55.6, 76.0 and 86.2.
template <int TYPE, bool EXACT, int R>
__device__ __forceinline__ void warp_generic(const MultArgs& M, int u, int q) {
  const int lane = threadIdx.x & 31;
  const int2* pairs = M.pairs + M.ptr[q];
  const int nt = (int)(M.ptr[q + 1] - M.ptr[q]);
  const int ndi = u ? u : M.prim_nsf[M.o_row[q]];
  const int ndo = u ? u : M.cover_nsf[M.o_cover[q]];    // type 1: nd_j ; type 2: nd_k
  const int ne = ndi * ndo;
  double acc[R];
  int n1[R], n2[R];                             // row and column of the lane's elements
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int e = min(lane + 32 * r, ne - 1);   // clamped: in-bounds reads
    n2[r] = e / ndi;
    n1[r] = e - ndi * n2[r];
    acc[r] = 0.0;
  }
  struct Term { const double *x, *b; int nk; };
  auto look_up = [&](int2 pr) {
    Term v;
    v.x = M.x + (u ? (int64_t)pr.x * (u * u) : M.x_elem[pr.x]);
    v.b = M.b + (u ? (int64_t)pr.y * (u * u) : M.b_elem[pr.y]);
    v.nk = u ? u : TYPE == 1 ? M.cover_nsf[M.x_cover[pr.x]] : M.cover_nsf[M.b_cover[pr.y]];
    return v;
  };
  Term next = {nullptr, nullptr, 0};
  int2 pn = make_int2(0, 0);
  if (nt > 0) next = look_up(__ldcs(pairs));
  if (nt > 1) pn = __ldcs(pairs + 1);
  for (int t = 0; t < nt; ++t) {
    const Term cur = next;
    if (t + 1 < nt) next = look_up(pn);
    if (t + 2 < nt) pn = __ldcs(pairs + t + 2);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (R > 1 && 32 * r >= ne) break;
      // type 1: a(n1, n) b(n, n2); type 2: c(n1, n) b(n2, n)
      const double *x = cur.x + n1[r], *b = cur.b + (TYPE == 1 ? cur.nk * n2[r] : n2[r]);
      double a = acc[r];
      if constexpr (R <= 2) {                   // blocks of at most K rows and columns: one batch of loads
        constexpr int K = R == 1 ? 5 : 8;
        double xv[K], bv[K];
#pragma unroll
        for (int n = 0; n < K; ++n)
          if (n < cur.nk) { xv[n] = __ldg(x + ndi * n); bv[n] = __ldg(b + (TYPE == 1 ? n : ndo * n)); }
#pragma unroll
        for (int n = 0; n < K; ++n)
          if (n < cur.nk) a = madd<EXACT>(a, xv[n], bv[n]);
      } else {
#pragma unroll 4
        for (int n = 0; n < cur.nk; ++n) a = madd<EXACT>(a, __ldg(x + ndi * n), __ldg(b + (TYPE == 1 ? n : ndo * n)));
      }
      acc[r] = a;
    }
  }
  double* O = M.out + M.o_elem[q];
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (lane + 32 * r < ne) O[lane + 32 * r] = acc[r];
}

template <int TYPE, bool EXACT, int R>
__global__ void __launch_bounds__(256) k_mult_generic(MultArgs M, int u) {
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q < M.n_out) warp_generic<TYPE, EXACT, R>(M, u, q);
}

// 4 x 4 blocks (SZ basis): 16 lanes per output block, one element per lane.  Each lane
// loads its operand row/column as two 16-byte vectors per block; blocks are 128 B aligned.
template <int TYPE, bool EXACT>
__global__ void __launch_bounds__(256) k_mult_nd4(MultArgs M) {
  int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 4, l = threadIdx.x & 15;
  if (g >= M.n_out) return;
  const int n1 = l & 3, m = l >> 2;   // element (n1, m) of the output block
  double acc = 0.0;
  const int64_t p0 = M.ptr[g], p1 = M.ptr[g + 1];
  for (int64_t t = p0; t < p1; ++t) {
    int2 pr = __ldcs(M.pairs + t);
    const double* X = M.x + M.x_elem[pr.x];
    const double* B = M.b + M.b_elem[pr.y];
    if (TYPE == 1) {
      // c(n1,m) += sum_n3 a(n1,n3) b(n3,m): a row is strided, b column contiguous
      double2 b01 = __ldg(reinterpret_cast<const double2*>(B + 4 * m));
      double2 b23 = __ldg(reinterpret_cast<const double2*>(B + 4 * m + 2));
      acc = madd<EXACT>(acc, __ldg(X + n1), b01.x);
      acc = madd<EXACT>(acc, __ldg(X + n1 + 4), b01.y);
      acc = madd<EXACT>(acc, __ldg(X + n1 + 8), b23.x);
      acc = madd<EXACT>(acc, __ldg(X + n1 + 12), b23.y);
    } else {
      // a(n1,m) += sum_n2 c(n1,n2) b(m,n2)
      acc = madd<EXACT>(acc, __ldg(X + n1), __ldg(B + m));
      acc = madd<EXACT>(acc, __ldg(X + n1 + 4), __ldg(B + m + 4));
      acc = madd<EXACT>(acc, __ldg(X + n1 + 8), __ldg(B + m + 8));
      acc = madd<EXACT>(acc, __ldg(X + n1 + 12), __ldg(B + m + 12));
    }
  }
  M.out[M.o_elem[g] + l] = acc;
}

// 4 x 4 blocks, one thread per output block with the whole block in registers: per triple
// the thread streams both operand blocks (8 + 8 16-byte loads) and does 64 multiply-adds,
// so the load/arithmetic ratio is 8x lower than with one lane per element.  Block b of a
// uniform 4 x 4 range starts at element 16 b.
template <int TYPE, bool EXACT>
__global__ void __launch_bounds__(128) k_mult_nd4_tpb(MultArgs M) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= M.n_out) return;
  double acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.0;
  const int64_t p0 = M.ptr[q], p1 = M.ptr[q + 1];
  for (int64_t t = p0; t < p1; ++t) {
    int2 pr = __ldcs(M.pairs + t);
    const double2* X2 = reinterpret_cast<const double2*>(M.x + 16 * (int64_t)pr.x);
    const double2* B2 = reinterpret_cast<const double2*>(M.b + 16 * (int64_t)pr.y);
    double x[16], b[16];
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      double2 xv = __ldg(X2 + v), bv = __ldg(B2 + v);
      x[2 * v] = xv.x; x[2 * v + 1] = xv.y;
      b[2 * v] = bv.x; b[2 * v + 1] = bv.y;
    }
    if (TYPE == 1) {
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n1 = 0; n1 < 4; ++n1) {
          double a = acc[n1 + 4 * m];
#pragma unroll
          for (int n3 = 0; n3 < 4; ++n3) a = madd<EXACT>(a, x[n1 + 4 * n3], b[n3 + 4 * m]);
          acc[n1 + 4 * m] = a;
        }
    } else {
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n1 = 0; n1 < 4; ++n1) {
          double a = acc[n1 + 4 * m];
#pragma unroll
          for (int n2 = 0; n2 < 4; ++n2) a = madd<EXACT>(a, x[n1 + 4 * n2], b[m + 4 * n2]);
          acc[n1 + 4 * m] = a;
        }
    }
  }
  double2* O2 = reinterpret_cast<double2*>(M.out + 16 * (int64_t)q);
#pragma unroll
  for (int v = 0; v < 8; ++v) __stcs(O2 + v, make_double2(acc[2 * v], acc[2 * v + 1]));
}

// 4 x 4 blocks, one thread per output block, the first operand's row staged in shared memory.
// A CTA owns up to 128 consecutive output blocks of one row i; every pair of those blocks reads
// its first operand from row i of that operand (A_ik for type 1, c_ij for type 2), so the row
// is copied into shared memory in chunks of CHUNK blocks with coalesced 16-byte loads, and each
// thread walks its pair list in order, taking the pairs whose operand lies in the current chunk
// (a pair list that goes back to an earlier chunk reads that block from global memory, so the
// order of the terms is never changed).  Only the B blocks come from L2 per pair.
template <int TYPE, bool EXACT, int CHUNK>
__global__ void __launch_bounds__(128) k_mult_nd4_rows(MultArgs M, const int4* __restrict__ tiles) {
  __shared__ double2 xs[CHUNK * 8];
  const int4 d = tiles[blockIdx.x];           // output blocks [d.x, d.y), operand row blocks [d.z, d.w)
  const int q = d.x + (int)threadIdx.x;
  int64_t t = 0, tend = 0;
  if (q < d.y) { t = M.ptr[q]; tend = M.ptr[q + 1]; }
  double acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.0;
  const double2* X2g = reinterpret_cast<const double2*>(M.x);
  const double2* B2g = reinterpret_cast<const double2*>(M.b);
  for (int c0 = d.z; c0 < d.w; c0 += CHUNK) {
    const int c1 = min(c0 + CHUNK, d.w);
    __syncthreads();
    for (int v = threadIdx.x; v < (c1 - c0) * 8; v += blockDim.x) xs[v] = __ldg(X2g + (int64_t)c0 * 8 + v);
    __syncthreads();
    while (t < tend) {
      const int2 pr = __ldcs(M.pairs + t);
      if (pr.x >= c1) break;
      double x[16], b[16];
      const double2* B2 = B2g + (int64_t)pr.y * 8;
      if (pr.x >= c0) {
        const double2* X2 = xs + (pr.x - c0) * 8;
#pragma unroll
        for (int v = 0; v < 8; ++v) { double2 xv = X2[v]; x[2 * v] = xv.x; x[2 * v + 1] = xv.y; }
      } else {
        const double2* X2 = X2g + (int64_t)pr.x * 8;
#pragma unroll
        for (int v = 0; v < 8; ++v) { double2 xv = __ldg(X2 + v); x[2 * v] = xv.x; x[2 * v + 1] = xv.y; }
      }
#pragma unroll
      for (int v = 0; v < 8; ++v) { double2 bv = __ldg(B2 + v); b[2 * v] = bv.x; b[2 * v + 1] = bv.y; }
      if (TYPE == 1) {
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int n1 = 0; n1 < 4; ++n1) {
            double a = acc[n1 + 4 * m];
#pragma unroll
            for (int n3 = 0; n3 < 4; ++n3) a = madd<EXACT>(a, x[n1 + 4 * n3], b[n3 + 4 * m]);
            acc[n1 + 4 * m] = a;
          }
      } else {
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int n1 = 0; n1 < 4; ++n1) {
            double a = acc[n1 + 4 * m];
#pragma unroll
            for (int n2 = 0; n2 < 4; ++n2) a = madd<EXACT>(a, x[n1 + 4 * n2], b[m + 4 * n2]);
            acc[n1 + 4 * m] = a;
          }
      }
      ++t;
    }
  }
  if (q < d.y) {
    double2* O2 = reinterpret_cast<double2*>(M.out + 16 * (int64_t)q);
#pragma unroll
    for (int v = 0; v < 8; ++v) __stcs(O2 + v, make_double2(acc[2 * v], acc[2 * v + 1]));
  }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 4 x 4 blocks, one thread per output block, operand blocks staged through shared memory by
// the whole warp.  A thread-per-block kernel that reads its own operand blocks issues 16-byte loads that touch 32
// different blocks per warp instruction, which saturates the L1 on wavefronts long before the FP64 pipe is busy.
// Here, per step, the warp copies the 32 (x, b) block pairs its lanes need with cp.async (8 consecutive lanes move
// one whole 128-byte block, 4 blocks per instruction), then every lane reads its two blocks and does its own
// 4 x 4 product in the reference order.  Output blocks are taken in `order` (descending pair count) so the lanes
// of a warp have pair lists of similar length.
// What bounds it: the 256 bytes that a pair moves from L2 (49 of the 64 bytes per SM and cycle) and about four L1
// wavefronts per pair.  The copies bypass the L1 (.cg): through it (.ca, or loads and shared-memory stores) the
// same kernel spends six.  Measured on LS.L -> LSL of the 512-atom cell (34.0 M pairs): 0.566 ms with .cg, 0.901
// with .ca, 1.009 with loads and stores; on the eight products of the LNV call 2.56, 3.96 and 4.58 ms.  One stage:
// the other 19 warps of an SM hide its latency, and a second stage (0.578 ms) costs L1, which the pair lists use
// (reading them two pairs at a time without it: 0.632 ms).
constexpr int kStageBytes = 64 * 128;    // one step of a warp: 32 X and 32 B blocks

// acc += the 4 x 4 product of the staged blocks x and b (both in registers), terms in the reference's order
template <int TYPE, bool EXACT>
__device__ __forceinline__ void nd4_mul_add(double (&acc)[16], const double (&x)[16], const double (&b)[16]) {
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n1 = 0; n1 < 4; ++n1) {
      double a = acc[n1 + 4 * m];
#pragma unroll
      for (int n = 0; n < 4; ++n) a = madd<EXACT>(a, x[n1 + 4 * n], TYPE == 1 ? b[n + 4 * m] : b[m + 4 * n]);
      acc[n1 + 4 * m] = a;
    }
}
// block `lane` of a stage: its 16-byte chunk v lies at chunk v ^ (lane & 7), so that the reads of eight lanes
// fall into different banks
__device__ __forceinline__ void nd4_read(double (&v)[16], const unsigned char* stage, int lane) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double2 d = *reinterpret_cast<const double2*>(stage + lane * 128 + ((k ^ (lane & 7)) << 4));
    v[2 * k] = d.x; v[2 * k + 1] = d.y;
  }
}

// One warp of the warp-staged 4 x 4 kernel: output slots [base, base + 32) of `order`, operand blocks
// staged through W (this warp's own shared memory).
template <int TYPE, bool EXACT>
__device__ __forceinline__ void warp_nd4_staged(const MultArgs& M, const int* __restrict__ order, int base, unsigned char* W) {
  const unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int slot = base + lane;
  const bool has = slot < M.n_out;
  const int q = has ? order[slot] : 0;
  const int2* pairs = M.pairs + (has ? M.ptr[q] : 0);
  const int nt = has ? (int)(M.ptr[q + 1] - M.ptr[q]) : 0;
  const int steps = __reduce_max_sync(kFull, nt);
  double acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.0;
  const double2* Xg = reinterpret_cast<const double2*>(M.x);
  const double2* Bg = reinterpret_cast<const double2*>(M.b);
  const int chunk = lane & 7;
  const uint32_t w0 = smem_addr(W);
  int2 pn = nt > 0 ? __ldcs(pairs) : make_int2(-1, -1);   // pair of the next step, loaded a step ahead
  for (int t = 0; t < steps; ++t) {
    const int2 pr = pn;
    pn = t + 1 < nt ? __ldcs(pairs + t + 1) : make_int2(-1, -1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int src = 4 * j + (lane >> 3);
      const int xb = __shfl_sync(kFull, pr.x, src);
      const int bb = __shfl_sync(kFull, pr.y, src);
      const uint32_t d = w0 + src * 128 + ((chunk ^ (src & 7)) << 4);
      if (xb >= 0) {
        cp_async16(d, Xg + (int64_t)xb * 8 + chunk);
        cp_async16(d + 4096, Bg + (int64_t)bb * 8 + chunk);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
    if (t < nt) {
      double x[16], b[16];
      nd4_read(x, W, lane);
      nd4_read(b, W + 4096, lane);
      nd4_mul_add<TYPE, EXACT>(acc, x, b);
    }
    __syncwarp();
  }
  if (has) {
    double2* O2 = reinterpret_cast<double2*>(M.out + 16 * (int64_t)q);
#pragma unroll
    for (int v = 0; v < 8; ++v) __stcs(O2 + v, make_double2(acc[2 * v], acc[2 * v + 1]));
  }
}

template <int TYPE, bool EXACT>
__global__ void __launch_bounds__(128, 5) k_mult_nd4_warp(MultArgs M, const int* __restrict__ order) {
  __shared__ __align__(128) unsigned char smem[4][kStageBytes];
  const int warp = threadIdx.x >> 5;
  const int base = (blockIdx.x * 4 + warp) * 32;
  if (base >= M.n_out) return;                  // whole warp
  warp_nd4_staged<TYPE, EXACT>(M, order, base, smem[warp]);
}

// Type 2, uniform 4 x 4 blocks: a(i, k) = sum over j in row k of B of c(i, j) b(k, j)^T.  All output blocks whose
// column atom is an image of one atom kh read the same row of B in the same order, so a warp takes 32 of them
// (one per lane) and walks that row: its B block is staged once per step and read by all lanes as a broadcast.
// That halves the bytes from L2 per pair and the shared-memory reads of B.  Two stages: these products have few
// output blocks, so an SM holds few warps.  Measured (512-atom cell, into the H range, 24064 output blocks): 0.325 ms
// against 0.473 for the warp-staged and 0.378 for the four-lanes-per-block kernel; into the L range (63664) 0.600
// against 0.601; three and four stages 0.766 and 0.878 there (the pair lists lose the L1).
// tile: (kh's row start in B, its end, first entry of trans_dest for the outputs, their number).
template <bool EXACT, int STAGES>
__global__ void __launch_bounds__(64) k_mult_nd4_row(MultArgs M, const int4* __restrict__ tiles, int n_tiles,
                                                     const int* __restrict__ trans_dest) {
  constexpr int kBytes = 4096 + 128;              // one step: 32 X blocks and the B block
  extern __shared__ __align__(128) unsigned char nd4_smem[];
  const unsigned kFull = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * 2 + warp;
  if (w >= n_tiles) return;                       // whole warp
  unsigned char* W = nd4_smem + warp * STAGES * kBytes;
  const int4 d = tiles[w];
  const bool has = lane < d.w;
  const int q = has ? trans_dest[d.z + lane] : 0;
  double acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.0;
  const double2* Xg = reinterpret_cast<const double2*>(M.x);
  const double2* Bg = reinterpret_cast<const double2*>(M.b);
  const int chunk = lane & 7;
  const uint32_t w0 = smem_addr(W);
  const int2* pairs = M.pairs + (has ? M.ptr[q] : 0);
  const int nt = has ? (int)(M.ptr[q + 1] - M.ptr[q]) : 0;
  int taken = 0;
  int2 pn = nt > 0 ? __ldg(pairs) : make_int2(-1, -1);      // the lane's next pair (its y is the B block)
  int2 pn2 = nt > 1 ? __ldg(pairs + 1) : make_int2(-1, -1);
  int eb = d.x;                                   // B block of the next step to stage
  unsigned act = 0;                               // bit s: the lane has a term in the step staged s steps ago
  auto issue = [&](int st) {
    const bool mine = pn.y == eb;                 // eb >= 0: never true past the list's end
    const int xl = mine ? pn.x : -1;
    act = act << 1 | (mine ? 1u : 0u);
    if (mine) {
      ++taken;
      pn = pn2;
      pn2 = taken + 1 < nt ? __ldg(pairs + taken + 1) : make_int2(-1, -1);
    }
    if (eb < d.y) {
      const uint32_t s = w0 + st * kBytes;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int src = 4 * j + (lane >> 3);
        const int xb = __shfl_sync(kFull, xl, src);
        if (xb >= 0) cp_async16(s + src * 128 + ((chunk ^ (src & 7)) << 4), Xg + (int64_t)xb * 8 + chunk);
      }
      if (lane < 8) cp_async16(s + 4096 + (lane << 4), Bg + (int64_t)eb * 8 + lane);
    }
    ++eb;
    cp_async_commit();
  };
  int st = 0;
#pragma unroll
  for (int k = 0; k + 1 < STAGES; ++k) issue(k);
  for (int e = d.x; e < d.y; ++e) {
    issue(st + STAGES - 1 >= STAGES ? st - 1 : st + STAGES - 1);
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    if (act >> (STAGES - 1) & 1) {
      const unsigned char* s = W + st * kBytes;
      double x[16], b[16];
      nd4_read(x, s, lane);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double2 v = *reinterpret_cast<const double2*>(s + 4096 + (k << 4));
        b[2 * k] = v.x; b[2 * k + 1] = v.y;
      }
      nd4_mul_add<2, EXACT>(acc, x, b);
    }
    __syncwarp();
    st = st + 1 == STAGES ? 0 : st + 1;
  }
  if (has) {
    double2* O2 = reinterpret_cast<double2*>(M.out + 16 * (int64_t)q);
#pragma unroll
    for (int v = 0; v < 8; ++v) __stcs(O2 + v, make_double2(acc[2 * v], acc[2 * v + 1]));
  }
}

// Uniform 4 x 4 blocks, one thread per output block, operand blocks staged by the bulk-copy (TMA)
// engine: every lane issues two 128-byte cp.async.bulk copies (its X and B blocks) into its slot of the warp's stage,
// whose mbarrier counts the bytes, so only the reads of the staged blocks go through the load/store
// pipe.  Three stages per warp keep the copies of the next two steps in flight.  Every wait is bounded
// (about a second; the error word is set and the warp stops).  The arithmetic is the warp-staged
// kernel's, in the same order: the same bits.  The copy engine bounds it: 68 M copies of 128 B in 2.59 ms on
// LS.L -> LSL of the 512-atom SZ cell, one per about 11 SM cycles (the warp-staged kernel takes 0.57 ms).  No rule
// chooses it.
constexpr int kBulkStages = 3;
constexpr int kBulkSlot = 144;            // bytes per staged block (128 + 16: conflict-free 16-byte reads)

__device__ __forceinline__ bool warp_bar_wait(unsigned long long* bar, uint32_t parity, int* err) {
  const uint32_t a = smem_addr(bar);
  uint64_t t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 63) == 0) {
      uint64_t t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (it == 0) t0 = t;
      else if (t - t0 > 1000000000ull) { *(volatile int*)err = 1; return false; }
    }
  }
}

template <int TYPE, bool EXACT>
__global__ void __launch_bounds__(128, 2) k_mult_nd4_bulk(MultArgs M, const int* __restrict__ order, int* err) {
  extern __shared__ __align__(128) unsigned char bulk_smem[];
  __shared__ unsigned long long bars[4][kBulkStages];
  const unsigned kFull = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int base = (blockIdx.x * 4 + warp) * 32;
  unsigned char* W = bulk_smem + (size_t)warp * kBulkStages * 64 * kBulkSlot;   // this warp's stages
  if (lane < kBulkStages)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bars[warp][lane])) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncwarp();
  if (base >= M.n_out) return;                  // whole warp (nothing waits on its barriers)
  const int slot = base + lane;
  const bool has = slot < M.n_out;
  const int q = has ? order[slot] : 0;
  const int64_t t = has ? M.ptr[q] : 0;
  const int64_t tend = has ? M.ptr[q + 1] : 0;
  double acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.0;
  const unsigned char* Xg = reinterpret_cast<const unsigned char*>(M.x);
  const unsigned char* Bg = reinterpret_cast<const unsigned char*>(M.b);
  // the copies of step s (the lane's pair t + s) into stage s % kBulkStages; lane 0 states the bytes
  // on the stage's barrier before any lane copies
  auto issue = [&](int s) {
    const int st = s % kBulkStages;
    const bool act = t + s < tend;
    const unsigned m = __ballot_sync(kFull, act);
    unsigned long long* bar = &bars[warp][st];
    if (lane == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(__popc(m) * 256u)
                   : "memory");
    __syncwarp();
    if (act) {
      const int2 pr = __ldcs(M.pairs + t + s);
      unsigned char* dst = W + ((size_t)st * 64 + 2 * lane) * kBulkSlot;
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 128, [%2];" ::"r"(
                       smem_addr(dst)),
                   "l"(Xg + (int64_t)pr.x * 128), "r"(smem_addr(bar))
                   : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 128, [%2];" ::"r"(
                       smem_addr(dst + kBulkSlot)),
                   "l"(Bg + (int64_t)pr.y * 128), "r"(smem_addr(bar))
                   : "memory");
    }
  };
  int issued = 0, done = 0;                     // steps whose copies were issued / which were consumed
  for (; issued < kBulkStages - 1; ++issued) issue(issued);
  for (int s = 0; __any_sync(kFull, t + s < tend); ++s) {
    issue(issued++);
    const int st = s % kBulkStages;
    const bool ok = __all_sync(kFull, warp_bar_wait(&bars[warp][st], (s / kBulkStages) & 1, err));
    if (!ok) break;
    if (t + s < tend) {
      const double2* X2 = reinterpret_cast<const double2*>(W + ((size_t)st * 64 + 2 * lane) * kBulkSlot);
      const double2* B2 = reinterpret_cast<const double2*>(W + ((size_t)st * 64 + 2 * lane + 1) * kBulkSlot);
      double x[16], b[16];
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const double2 xv = X2[v], bv = B2[v];
        x[2 * v] = xv.x; x[2 * v + 1] = xv.y;
        b[2 * v] = bv.x; b[2 * v + 1] = bv.y;
      }
      if (TYPE == 1) {
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int n1 = 0; n1 < 4; ++n1) {
            double a = acc[n1 + 4 * m];
#pragma unroll
            for (int n3 = 0; n3 < 4; ++n3) a = madd<EXACT>(a, x[n1 + 4 * n3], b[n3 + 4 * m]);
            acc[n1 + 4 * m] = a;
          }
      } else {
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int n1 = 0; n1 < 4; ++n1) {
            double a = acc[n1 + 4 * m];
#pragma unroll
            for (int n2 = 0; n2 < 4; ++n2) a = madd<EXACT>(a, x[n1 + 4 * n2], b[m + 4 * n2]);
            acc[n1 + 4 * m] = a;
          }
      }
    }
    done = s + 1;
    __syncwarp();                               // the stage is read before step s + kBulkStages refills it
  }
  // steps issued but not consumed (the empty steps after the last pair, or the copies in flight when a
  // wait ran out): wait for them (bounded) before the CTA's shared memory is released
  for (int s = done; s < issued; ++s) warp_bar_wait(&bars[warp][s % kBulkStages], (s / kBulkStages) & 1, err);
  if (has) {
    double2* O2 = reinterpret_cast<double2*>(M.out + 16 * (int64_t)q);
#pragma unroll
    for (int v = 0; v < 8; ++v) __stcs(O2 + v, make_double2(acc[2 * v], acc[2 * v + 1]));
  }
}

// Uniform 4 x 4 blocks, four lanes per output block: lane m of a quad owns column m of the block
// (elements n1 + 4m, n1 = 0..3).  The quad copies the two blocks of a pair into its slots of a ring of
// STAGES stages (cp.async, two 16-byte chunks of each block per lane), all four lanes read the X block as a
// broadcast and each lane its column of B.  Four times the lanes of k_mult_nd4_warp, and STAGES - 1 pairs in
// flight per quad, for products with few output blocks, whose time is the latency of their lists' steps.
// Measured with 3, 4 and 6 stages: 64 atoms into the L range (1862 output blocks, 167 pairs each) 37.0, 35.0 and
// 33.4 us (91 for the warp-staged kernel, 105 for one lane per element), 216 atoms L.S -> LS (115274) 23.0, 24.8
// and 26.8 us (31.0 warp-staged).  Without the ring the 512-atom product into the H range took 0.545 ms; now 0.389.
// Every element keeps the order of its terms, so the results are the same bits.
template <int TYPE, bool EXACT, int STAGES>
__global__ void __launch_bounds__(128) k_mult_nd4_quad(MultArgs M, const int* __restrict__ order) {
  __shared__ __align__(128) unsigned char smem[4][STAGES][8 * 256];   // per quad: the X block, then the B block
  const unsigned kFull = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qd = lane >> 2, m = lane & 3;
  const int base = (blockIdx.x * 4 + warp) * 8;  // first output slot of this warp
  if (base >= M.n_out) return;                   // whole warp
  const int slot = base + qd;
  const bool has = slot < M.n_out;
  const int q = has ? order[slot] : 0;
  const int2* pairs = M.pairs + (has ? M.ptr[q] : 0);
  const int nt = has ? (int)(M.ptr[q + 1] - M.ptr[q]) : 0;
  const int steps = __reduce_max_sync(kFull, nt);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const double2* Xg = reinterpret_cast<const double2*>(M.x);
  const double2* Bg = reinterpret_cast<const double2*>(M.b);
  // chunk v of a block lies at chunk v ^ qd: the eight quads' reads of one chunk fall into different banks
  const int c0 = (m ^ qd) << 4, c1 = ((m + 4) ^ qd) << 4;
  int issued = 0;
  int2 pn = nt > 0 ? __ldcs(pairs) : make_int2(0, 0);    // the next pair to copy, loaded a step ahead
  auto issue = [&](int st) {
    if (issued < nt) {
      const uint32_t d = smem_addr(smem[warp][st]) + qd * 256;
      const double2 *xs = Xg + (int64_t)pn.x * 8 + m, *bs = Bg + (int64_t)pn.y * 8 + m;
      cp_async16(d + c0, xs);
      cp_async16(d + c1, xs + 4);
      cp_async16(d + 128 + c0, bs);
      cp_async16(d + 128 + c1, bs + 4);
      if (issued + 1 < nt) pn = __ldcs(pairs + issued + 1);
    }
    ++issued;
    cp_async_commit();
  };
  int st = 0;
#pragma unroll
  for (int k = 0; k + 1 < STAGES; ++k) issue(k);
  for (int t = 0; t < steps; ++t) {
    issue(st == 0 ? STAGES - 1 : st - 1);
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    if (t < nt) {
      const unsigned char* X = smem[warp][st] + qd * 256;
      const unsigned char* B = X + 128;
      double x[16], bc[4];
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const double2 xv = *reinterpret_cast<const double2*>(X + ((v ^ qd) << 4));
        x[2 * v] = xv.x; x[2 * v + 1] = xv.y;
      }
      if (TYPE == 1) {
        // B[n3 + 4m], n3 = 0..3: the four contiguous values of column m
        const double2 u = *reinterpret_cast<const double2*>(B + (((2 * m) ^ qd) << 4));
        const double2 v = *reinterpret_cast<const double2*>(B + (((2 * m + 1) ^ qd) << 4));
        bc[0] = u.x; bc[1] = u.y; bc[2] = v.x; bc[3] = v.y;
      } else {
        // B[m + 4 n2], n2 = 0..3
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2)
          bc[n2] = *reinterpret_cast<const double*>(B + (((2 * n2 + (m >> 1)) ^ qd) << 4) + ((m & 1) << 3));
      }
      // type 1: acc[n1] += sum_n3 x[n1 + 4 n3] B[n3 + 4m]; type 2: acc[n1] += sum_n2 x[n1 + 4 n2] B[m + 4 n2]
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) {
        double a = acc[n1];
#pragma unroll
        for (int n = 0; n < 4; ++n) a = madd<EXACT>(a, x[n1 + 4 * n], bc[n]);
        acc[n1] = a;
      }
    }
    __syncwarp();                                // the stage is read before the next issue() refills it
    st = st + 1 == STAGES ? 0 : st + 1;
  }
  if (has) {
    double2* O2 = reinterpret_cast<double2*>(M.out + 16 * (int64_t)q) + 2 * m;
    __stcs(O2, make_double2(acc[0], acc[1]));
    __stcs(O2 + 1, make_double2(acc[2], acc[3]));
  }
}

// Any block sizes up to 16 (DZP 13 x 13, mixed SZ/DZP): LPB lanes per output block (8: four blocks per warp,
// lane l owns columns l and l + 8; 16: two blocks per warp, one column per lane), every row of those columns in
// the lane's registers.  The group stages the two operand blocks of a pair in shared memory with cp.async; X
// with its columns padded to an even length, so that two row values are one 16-byte read that all lanes of a
// group share, B in its stored layout (a block of odd size starts on an 8-byte boundary: its copy keeps the
// source's 8-byte phase and moves the odd first or last element alone).  Buffers are an odd multiple of 32
// bytes long, so the groups' broadcast reads fall into different banks.  The order of the terms of every
// element is unchanged.
//
// What bounds it: the FP64 pipe and the shared-memory reads.  A 13 x 13 pair is 2 x 13^3 FP64 instructions on
// 13 of 16 columns (84 SM cycles); a 16-byte read takes two L1 wavefronts even as a broadcast, so with LPB = 8 a
// pair costs about 88 wavefronts, with LPB = 16 129.  Against it LPB = 8 needs twice the shared memory per warp.
// Measured (64-atom DZP cell, LS.L -> LSL, 147794 output blocks, 4.2 M pairs, reference rounding; TFLOP/s): LPB 8
// with one stage 10.5, with two 9.7 and three 9.1 (fewer warps per SM); LPB 16 with one 9.3, two 9.2, four 7.9;
// one block per warp with 4 x 2 tiles and operands read from global memory 3.4.  With many warps per SM the
// other warps hide a stage's latency, so one stage is best.  With few output blocks (3008, type 2 into the H
// range) LPB 16 with two stages runs at 7.4 against 6.2: twice the warps, and the next pair's copies in flight.
// The two are equal near 8000 output blocks (8.6).
// U: the block size when the whole system has one, else 0.  MAXND: no block is larger.
template <int MAXND, int LPB, int STAGES>
struct GroupShape {
  static constexpr int kBlocks = 32 / LPB;                            // output blocks per warp
  // bytes of one staged block, odd multiples of 32: X with its columns padded to an even length, B as stored
  static constexpr int kStrideX = 32 * (((MAXND + 1) / 2 * 2 * MAXND * 8 + 31) / 32 | 1);
  static constexpr int kStrideB = 32 * ((MAXND * MAXND * 8 + 8 + 31) / 32 | 1);
  static constexpr int kStage = kBlocks * (kStrideX + kStrideB);      // the X blocks, then the B blocks
  static constexpr int kWarpBytes = STAGES * kStage;
  static_assert(2 * kWarpBytes <= 48 * 1024, "two warps fit the shared memory that every launch may take");
};

// n doubles at src (8-byte aligned) to the 16-byte aligned slot dst, by the LPB lanes l of a group; the data
// starts at dst + 8 when src is not 16-byte aligned.  Reads no byte outside [src, src + n).
template <int U, int LPB>
__device__ __forceinline__ void group_copy(uint32_t dst, const double* src, int n, int l) {
  const int sh = (int)(((uintptr_t)src >> 3) & 1);
  const int chunks = (n - sh) >> 1;
  const double* s16 = src + sh;
  const uint32_t d16 = dst + 16 * sh;
  if constexpr (U > 0) {
    constexpr int kIter = (U * U / 2 + LPB - 1) / LPB;
#pragma unroll
    for (int v = 0; v < kIter; ++v)
      if (l + LPB * v < chunks) cp_async16(d16 + 16 * (l + LPB * v), s16 + 2 * (l + LPB * v));
  } else {
    for (int v = l; v < chunks; v += LPB) cp_async16(d16 + 16 * v, s16 + 2 * v);
  }
  if (l == LPB - 2 && sh) cp_async8(dst + 8, src);
  if (l == LPB - 1 && ((n - sh) & 1)) cp_async8(dst + 8 * (sh + n - 1), src + n - 1);
}

// The X block (rows x cols, n = rows * cols doubles at src) to the slot dst with its columns ld doubles apart
// (rows rounded up to even), so that two row values are one 16-byte shared-memory read.  magic: 65536 / rows + 1.
template <int U, int LPB>
__device__ __forceinline__ void group_copy_columns(uint32_t dst, const double* src, int n, int rows, int magic, int l) {
  if constexpr (U > 0) {
    constexpr int kIter = (U * U + LPB - 1) / LPB;
#pragma unroll
    for (int v = 0; v < kIter; ++v) {
      const int e = l + LPB * v;
      if (e < U * U) cp_async8(dst + 8 * (e + (U & 1) * (e / U)), src + e);
    }
  } else {
    const int pad = rows & 1;
    for (int e = l; e < n; e += LPB) cp_async8(dst + 8 * (e + pad * ((e * magic) >> 16)), src + e);
  }
}

// One pair's arithmetic: acc[r][h] (row r, column c[h]) += sum over n < nk.
template <int TYPE, bool EXACT, int U, int R, bool FULL, int H>
__device__ __forceinline__ void group_compute(const double2* __restrict__ X, const double* __restrict__ B, int ndi, int ndo,
                                              int nk, const int (&c)[H], int cols, double (&acc)[R][H]) {
  const int half = FULL ? (R + 1) / 2 : (ndi + 1) >> 1;           // double2 per column of X
  auto step = [&](int n) {
    double2 x[(R + 1) / 2];
    double b[H];
#pragma unroll
    for (int r = 0; r < (R + 1) / 2; ++r) x[r] = X[(FULL ? r : min(r, half - 1)) + half * n];
#pragma unroll
    for (int h = 0; h < H; ++h)
      if (h < cols) b[h] = TYPE == 1 ? B[n + nk * c[h]] : B[c[h] + ndo * n];
#pragma unroll
    for (int h = 0; h < H; ++h)
      if (h < cols) {
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r][h] = madd<EXACT>(acc[r][h], r & 1 ? x[r / 2].y : x[r / 2].x, b[h]);
      }
  };
  if constexpr (U > 0) {
#pragma unroll
    for (int n = 0; n < U; ++n) step(n);
  } else {
#pragma unroll 2
    for (int n = 0; n < nk; ++n) step(n);
  }
}

// One warp: output slots [base, base + 32 / LPB) of `order`; W: this warp's shared memory (STAGES stages).
// R: rows of the register tile; FULL: every block of the warp has exactly R rows.
template <int TYPE, bool EXACT, int U, int MAXND, int LPB, int STAGES, int R, bool FULL>
__device__ __forceinline__ void warp_group_rows(const MultArgs& M, const int* __restrict__ order, int base, unsigned char* W) {
  using Q = GroupShape<MAXND, LPB, STAGES>;
  constexpr int H = 16 / LPB;                      // columns per lane
  const unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31, g = lane / LPB, l = lane % LPB;
  const bool has = base + g < M.n_out;
  const int q = has ? order[base + g] : 0;
  const int ndi = FULL ? R : M.prim_nsf[M.o_row[q]];
  const int ndo = U > 0 ? U : M.cover_nsf[M.o_cover[q]];     // type 1: nd_j ; type 2: nd_k
  int c[H];
#pragma unroll
  for (int h = 0; h < H; ++h) c[h] = min(l + LPB * h, ndo - 1);   // clamped: in-bounds reads
  const int cols = H == 1 || (U > 0 ? U > LPB : __any_sync(kFull, ndo > LPB)) ? H : 1;
  const int2* pairs = M.pairs + (has ? M.ptr[q] : 0);
  const int nt = has ? (int)(M.ptr[q + 1] - M.ptr[q]) : 0;       // a list is no longer than a row: fits 32 bits
  const int steps = __reduce_max_sync(kFull, nt);
  double acc[R][H];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int h = 0; h < H; ++h) acc[r][h] = 0.0;
  const uint32_t w0 = smem_addr(W);
  const int magic = U > 0 ? 0 : 65536 / ndi + 1;   // e / ndi = e * magic >> 16 for e < 256, ndi <= 16
  // operand addresses and inner dimension of a pair; looked up one step before its copies are issued
  struct Term { const double *x, *b; int nk; };
  auto look_up = [&](int2 pr) {
    Term v;
    v.x = M.x + (U > 0 ? (int64_t)pr.x * (U * U) : M.x_elem[pr.x]);
    v.b = M.b + (U > 0 ? (int64_t)pr.y * (U * U) : M.b_elem[pr.y]);
    v.nk = U > 0 ? U : (TYPE == 1 ? M.cover_nsf[M.x_cover[pr.x]] : M.cover_nsf[M.b_cover[pr.y]]);
    return v;
  };
  Term next = {nullptr, nullptr, 0};               // pair `issued`
  int2 pn = make_int2(0, 0);                       // pair `issued + 1`
  if (nt > 0) next = look_up(__ldcs(pairs));
  if (nt > 1) pn = __ldcs(pairs + 1);
  int issued = 0, slot = 0;                        // pairs whose copies were issued, and the stage of the next one
  int meta[STAGES];                                // 2 nk + the 8-byte phase of the B copy, per stage in flight
  auto issue = [&]() {
    int mt = 0;
    if (issued < nt) {
      const uint32_t d = w0 + slot * Q::kStage;
      mt = 2 * next.nk + (int)(((uintptr_t)next.b >> 3) & 1);
      group_copy_columns<U, LPB>(d + g * Q::kStrideX, next.x, ndi * next.nk, ndi, magic, l);
      group_copy<U, LPB>(d + Q::kBlocks * Q::kStrideX + g * Q::kStrideB, next.b, next.nk * ndo, l);
      if (issued + 1 < nt) next = look_up(pn);
      if (issued + 2 < nt) pn = __ldcs(pairs + issued + 2);
    }
    cp_async_commit();
    ++issued;
    slot = slot + 1 == STAGES ? 0 : slot + 1;
#pragma unroll
    for (int k = 0; k + 1 < STAGES; ++k) meta[k] = meta[k + 1];
    meta[STAGES - 1] = mt;
  };
#pragma unroll
  for (int k = 0; k < STAGES; ++k) meta[k] = 0;
#pragma unroll
  for (int k = 0; k + 1 < STAGES; ++k) issue();
  int st = 0;
  for (int t = 0; t < steps; ++t) {
    issue();
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    if (t < nt) {
      const unsigned char* s = W + st * Q::kStage;
      const double2* X = reinterpret_cast<const double2*>(s + g * Q::kStrideX);
      const double* B = reinterpret_cast<const double*>(s + Q::kBlocks * Q::kStrideX + g * Q::kStrideB) + (meta[0] & 1);
      group_compute<TYPE, EXACT, U, R, FULL, H>(X, B, ndi, ndo, meta[0] >> 1, c, cols, acc);
    }
    __syncwarp();                                  // the stage is read before the next issue() refills it
    st = st + 1 == STAGES ? 0 : st + 1;
  }
  // results through shared memory (the staging buffers are free: no copy is in flight), so that a group
  // writes its block to consecutive addresses
  double* O = reinterpret_cast<double*>(W + g * Q::kStrideX);
#pragma unroll
  for (int h = 0; h < H; ++h)
    if (l + LPB * h < ndo) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (FULL || r < ndi) O[r + ndi * (l + LPB * h)] = acc[r][h];
    }
  __syncwarp();
  if (has) {
    double* D = M.out + (U > 0 ? (int64_t)q * (U * U) : M.o_elem[q]);
    for (int e = l; e < ndi * ndo; e += LPB) __stcs(D + e, O[e]);
  }
  __syncwarp();
}

template <int TYPE, bool EXACT, int U, int MAXND, int LPB, int STAGES>
__device__ __forceinline__ void warp_group(const MultArgs& M, const int* __restrict__ order, int base, unsigned char* W) {
  if constexpr (U > 0) {
    warp_group_rows<TYPE, EXACT, U, MAXND, LPB, STAGES, U, true>(M, order, base, W);
  } else {
    // several sizes: a warp whose blocks all have four rows, or all MAXND, runs a tile of exactly that height
    // (the order keeps blocks of one row count together)
    const int s = min(base + (threadIdx.x & 31) / LPB, M.n_out - 1);
    const int ndi = M.prim_nsf[M.o_row[order[s]]];
    if (__all_sync(0xffffffffu, ndi == 4)) warp_group_rows<TYPE, EXACT, 0, MAXND, LPB, STAGES, 4, true>(M, order, base, W);
    else if (__all_sync(0xffffffffu, ndi == MAXND)) warp_group_rows<TYPE, EXACT, 0, MAXND, LPB, STAGES, MAXND, true>(M, order, base, W);
    else warp_group_rows<TYPE, EXACT, 0, MAXND, LPB, STAGES, MAXND, false>(M, order, base, W);
  }
}

template <int TYPE, bool EXACT, int U, int MAXND, int LPB, int STAGES>
__global__ void __launch_bounds__(64) k_mult_group(MultArgs M, const int* __restrict__ order) {
  extern __shared__ __align__(128) unsigned char group_smem[];
  using Q = GroupShape<MAXND, LPB, STAGES>;
  const int warp = threadIdx.x >> 5;
  const int base = (blockIdx.x * 2 + warp) * Q::kBlocks;
  if (base >= M.n_out) return;                  // whole warp
  warp_group<TYPE, EXACT, U, MAXND, LPB, STAGES>(M, order, base, group_smem + warp * Q::kWarpBytes);
}

// FP64 on the tensor cores (DMMA, mma.sync.m8n8k4.f64): one warp per output block, the block padded to 16 x 16 as
// 2 x 2 tiles of 8 x 8.  Per step of four contraction indices a lane reads one element of each first-operand row
// tile (row g = lane / 4, index t = lane % 4 of the step) and one of each B column tile (index t, column g), zeros
// outside the blocks, and the warp issues four MMAs; C/D hold rows g, columns 2t and 2t + 1 of each tile.  The
// terms of an element are summed in FP64 by the tensor cores in the blocks' order, four at a time, so the result
// differs from the reference kernel's separate multiply and add in rounding only (about 1e-16 of sum |a||b|).
//
// Four pairs at a time are staged in shared memory (cp.async, eight lanes per pair) and their contractions run
// as one: the steps cross from one pair to the next, so four 13 x 13 pairs take 13 steps instead of 4 x 4 and
// the order of the terms stays.  What bounds it: the FP64 tensor pipe (52 MMAs per four pairs, 52 SM cycles a
// pair), the shared-memory reads of the fragments (33 L1 wavefronts a pair and about as many to stage it) and the
// 2.7 KB a pair moves from L2 (42 cycles).  One stage: the other warps of the SM hide its latency.
// Measured (216-atom DZP cell, SLS = LS.S, 3.4 M pairs): 1.23 ms = 12.0 TFLOP/s, tensor pipe 50 % busy, L2 at 66 % of
// its throughput; operands read straight from global memory, one pair at a time, 1.71 ms. The eight products of
// an LNV call 25.1 -> 19.8 ms.
__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <int TYPE, int U, int MAXND>
__global__ void __launch_bounds__(64) k_mult_dmma(MultArgs M, const int* __restrict__ order) {
  constexpr int kStride = GroupShape<MAXND, 8, 1>::kStrideB;       // bytes of one staged block
  __shared__ __align__(128) unsigned char smem[2][8 * kStride];    // per warp: four X and four B blocks
  const unsigned kFull = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = blockIdx.x * 2 + warp;
  if (slot >= M.n_out) return;                    // whole warp
  const int q = order ? order[slot] : slot;      // null: the stored order
  const int g = lane >> 2, t = lane & 3;          // fragment row / column and contraction index
  const int gp = lane >> 3, l = lane & 7;         // staging: pair and lane of its group
  unsigned char* W = smem[warp];
  const int ndi = U > 0 ? U : M.prim_nsf[M.o_row[q]];
  const int ndo = U > 0 ? U : M.cover_nsf[M.o_cover[q]];     // type 1: nd_j ; type 2: nd_k
  const bool r0 = U >= 8 || g < ndi, r1 = g + 8 < ndi, c0 = U >= 8 || g < ndo, c1 = g + 8 < ndo;
  const bool rt = ndi > 8, ct = ndo > 8;          // a second row / column tile
  double acc[2][2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int2* pairs = M.pairs + M.ptr[q];
  const int nt = (int)(M.ptr[q + 1] - M.ptr[q]);
  const uint32_t w0 = smem_addr(W);
  // the group's pair of the next round with its addresses looked up, and the pair of the round after that
  struct Term { const double *x, *b; int nk; };
  auto look_up = [&](int2 pr) {
    Term v = {nullptr, nullptr, 0};
    if (pr.x >= 0) {
      v.x = M.x + (U > 0 ? (int64_t)pr.x * (U * U) : M.x_elem[pr.x]);
      v.b = M.b + (U > 0 ? (int64_t)pr.y * (U * U) : M.b_elem[pr.y]);
      v.nk = U > 0 ? U : (TYPE == 1 ? M.cover_nsf[M.x_cover[pr.x]] : M.cover_nsf[M.b_cover[pr.y]]);
    }
    return v;
  };
  auto pair_of = [&](int k) { return k < nt ? __ldcs(pairs + k) : make_int2(-1, -1); };
  Term next = look_up(pair_of(gp));
  int2 pn = pair_of(4 + gp);
  for (int t0 = 0; t0 < nt; t0 += 4) {
    const int nk = next.nk;                       // 0 past the list's end
    const bool px = ((uintptr_t)next.x >> 3) & 1, pb = ((uintptr_t)next.b >> 3) & 1;   // 8-byte phases of the copies
    if (nk > 0) {
      group_copy<U, 8>(w0 + gp * kStride, next.x, ndi * nk, l);
      group_copy<U, 8>(w0 + (4 + gp) * kStride, next.b, nk * ndo, l);
    }
    next = look_up(pn);
    pn = pair_of(t0 + 8 + gp);
    cp_async_commit();
    const unsigned mx = __ballot_sync(kFull, px), mb = __ballot_sync(kFull, pb);
    // contraction offsets of the pairs
    const int n0 = U > 0 ? U : __shfl_sync(kFull, nk, 0), n1 = U > 0 ? U : __shfl_sync(kFull, nk, 8),
              n2 = U > 0 ? U : __shfl_sync(kFull, nk, 16), n3 = U > 0 ? U : __shfl_sync(kFull, nk, 24);
    const int o1 = n0, o2 = o1 + n1, o3 = o2 + n2;
    const int K = U > 0 ? U * min(4, nt - t0) : o3 + n3;
    cp_async_wait<0>();
    __syncwarp();
    auto step = [&](int ks, bool all) {
      const int kk = 4 * ks + t;
      const int p = U > 0 ? kk / (U > 0 ? U : 1) : (kk >= o1) + (kk >= o2) + (kk >= o3);
      const int off = U > 0 ? p * U : p == 0 ? 0 : p == 1 ? o1 : p == 2 ? o2 : o3;
      const int n = kk - off;
      const bool in = all || kk < K;
      const double* X = reinterpret_cast<const double*>(W + p * kStride) + ((mx >> (8 * p)) & 1) + g + ndi * n;
      const int np = U > 0 ? U : p == 0 ? n0 : p == 1 ? n1 : p == 2 ? n2 : n3;
      const double* B = reinterpret_cast<const double*>(W + (4 + p) * kStride) + ((mb >> (8 * p)) & 1) +
                        (TYPE == 1 ? n + np * g : g + ndo * n);
      const double a0 = in && r0 ? X[0] : 0.0, a1 = in && r1 ? X[8] : 0.0;
      const double b0 = in && c0 ? B[0] : 0.0, b1 = in && c1 ? B[TYPE == 1 ? 8 * np : 8] : 0.0;
      dmma_8x8x4(acc[0][0], a0, b0);
      if (ct) dmma_8x8x4(acc[0][1], a0, b1);
      if (rt) dmma_8x8x4(acc[1][0], a1, b0);
      if (rt && ct) dmma_8x8x4(acc[1][1], a1, b1);
    };
    if (U > 0 && K == 4 * U) {
#pragma unroll
      for (int ks = 0; ks < U; ++ks) step(ks, true);
    } else {
      for (int ks = 0; 4 * ks < K; ++ks) step(ks, false);
    }
    __syncwarp();                                 // the blocks are read before the next round replaces them
  }
  // results through shared memory, so that the block is written along memory
  double* O = reinterpret_cast<double*>(W);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = 8 * i + g, c = 8 * j + 2 * t + e;
        if (r < ndi && c < ndo) O[r + ndi * c] = acc[i][j][e];
      }
  __syncwarp();
  double* D = M.out + (U > 0 ? (int64_t)q * (U * U) : M.o_elem[q]);
  for (int e = lane; e < ndi * ndo; e += 32) __stcs(D + e, O[e]);
}

// The same MMAs for short lists: one warp per output block in the stored order, one pair at a time, the operands read
// straight from the block storage into fragments (the next pair's while the current one's MMAs run), no shared memory.
// What bounds it is that chain of loads; it is the faster one where a list is a round or two long (dmma_short).
template <int TYPE>
__device__ __forceinline__ void dmma_load_pair(const MultArgs& M, int2 pr, int ndi, int ndo, int g, int t,
                                               double (&av)[4][2], double (&bv)[4][2], int& nks) {
  const double* X = M.x + M.x_elem[pr.x];
  const double* B = M.b + M.b_elem[pr.y];
  const int nk = TYPE == 1 ? M.cover_nsf[M.x_cover[pr.x]] : M.cover_nsf[M.b_cover[pr.y]];
  nks = (nk + 3) >> 2;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    const int n = 4 * ks + t;
    const bool in = n < nk;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = 8 * h + g;                     // row of the first operand's fragment, column of B's
      av[ks][h] = in && e < ndi ? __ldg(X + e + ndi * n) : 0.0;
      bv[ks][h] = in && e < ndo ? __ldg(TYPE == 1 ? B + n + nk * e : B + e + ndo * n) : 0.0;
    }
  }
}

template <int TYPE>
__global__ void __launch_bounds__(128) k_mult_dmma_short(MultArgs M) {
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= M.n_out) return;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int2* pairs = M.pairs + M.ptr[q];
  const int nt = (int)(M.ptr[q + 1] - M.ptr[q]);
  const int ndi = M.prim_nsf[M.o_row[q]];
  const int ndo = M.cover_nsf[M.o_cover[q]];     // type 1: nd_j ; type 2: nd_k
  const bool rt = ndi > 8, ct = ndo > 8;         // a second row / column tile
  double acc[2][2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  double av[4][2], bv[4][2];
  int nks = 0;
  if (nt > 0) dmma_load_pair<TYPE>(M, __ldcs(pairs), ndi, ndo, g, t, av, bv, nks);
  for (int p = 0; p < nt; ++p) {
    double nav[4][2], nbv[4][2];
    int nnks = 0;
    if (p + 1 < nt) dmma_load_pair<TYPE>(M, __ldcs(pairs + p + 1), ndi, ndo, g, t, nav, nbv, nnks);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      if (ks < nks) {
        dmma_8x8x4(acc[0][0], av[ks][0], bv[ks][0]);
        if (ct) dmma_8x8x4(acc[0][1], av[ks][0], bv[ks][1]);
        if (rt) dmma_8x8x4(acc[1][0], av[ks][1], bv[ks][0]);
        if (rt && ct) dmma_8x8x4(acc[1][1], av[ks][1], bv[ks][1]);
      }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int h = 0; h < 2; ++h) { av[ks][h] = nav[ks][h]; bv[ks][h] = nbv[ks][h]; }
    nks = nnks;
  }
  double* O = M.out + M.o_elem[q];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = 8 * i + g, c = 8 * j + 2 * t + e;
        if (r < ndi && c < ndo) O[r + ndi * c] = acc[i][j][e];
      }
}

// Many independent products in one persistent launch (the concatenation of their output-block
// lists): every warp takes work units u = warp id, warp id + warps in the grid, ...; a unit is 32
// output slots of a uniform 4 x 4 product (the warp-staged kernel) or two output blocks of any other product (the group
// kernel with 16 lanes per block), or one output block where all products are of small blocks (the generic kernel).  Each output block is computed by exactly the operations
// of the single-product kernels, so the results are the same bits as separate launches.  The product table
// travels in the kernel's parameters (no host-to-device copy before the launch).  Eight systems of 64 to 300 atoms
// (1.98 GFLOP): 0.284 ms, against 0.684 ms with one output block per warp and register tiles of 4 x 2.
struct BatchProduct {
  MultArgs M;
  const int* order;                // output blocks by descending pair count
  int kind;                        // bit 0: type 2, bit 1: exact rounding, bits 2..: kBatchNd4, ...
  int u;                           // the block size when the whole system has one, else 0
};
enum { kBatchNd4 = 0, kBatchU13 = 4, kBatchMax13 = 8, kBatchMax16 = 12 };
constexpr int kBatchMax = 96;      // products per launch (the table stays within the 32 KB parameter space)
struct BatchParams {
  int n_prod;
  int unit_off[kBatchMax + 1];     // first work unit of each product; unit_off[n_prod] = all units
  BatchProduct prods[kBatchMax];
};
static_assert(sizeof(BatchParams) < 32000, "batched product table exceeds the kernel parameter space");

constexpr int kBatchWarpBytes = kStageBytes + 256;    // the larger of the two kernels' staging areas
static_assert(GroupShape<13, 16, 1>::kWarpBytes <= kBatchWarpBytes && GroupShape<16, 16, 1>::kWarpBytes <= kBatchWarpBytes,
              "batched warps share one staging area");

template <int TYPE, bool EXACT, bool SMALL>
__device__ __forceinline__ void batch_unit(const BatchProduct& P, int family, int unit, unsigned char* W) {
  if constexpr (SMALL) {
    warp_generic<TYPE, EXACT, 1>(P.M, P.u, unit);
  } else if (family == kBatchNd4) {
    warp_nd4_staged<TYPE, EXACT>(P.M, P.order, unit * 32, W);
  } else if (family == kBatchU13) {
    warp_group<TYPE, EXACT, 13, 13, 16, 1>(P.M, P.order, unit * 2, W);
  } else if (family == kBatchMax13) {
    warp_group<TYPE, EXACT, 0, 13, 16, 1>(P.M, P.order, unit * 2, W);
  } else {
    warp_group<TYPE, EXACT, 0, 16, 16, 1>(P.M, P.order, unit * 2, W);
  }
}

// SMALL: every product is of small blocks (batch_of_small_blocks)
template <bool SMALL>
__global__ void __launch_bounds__(128, 4) k_mult_batch(const __grid_constant__ BatchParams B) {
  __shared__ __align__(128) unsigned char smem[4][SMALL ? 16 : kBatchWarpBytes];
  const int warp = threadIdx.x >> 5;
  const int n_units = B.unit_off[B.n_prod];
  for (int u = blockIdx.x * 4 + warp; u < n_units; u += gridDim.x * 4) {
    int lo = 0, hi = B.n_prod - 1;               // product of unit u: last p with unit_off[p] <= u
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (B.unit_off[mid] <= u) lo = mid; else hi = mid - 1;
    }
    const BatchProduct& P = B.prods[lo];
    const int family = P.kind & ~3, unit = u - B.unit_off[lo];
    switch (P.kind & 3) {
      case 0: batch_unit<1, false, SMALL>(P, family, unit, smem[warp]); break;
      case 1: batch_unit<2, false, SMALL>(P, family, unit, smem[warp]); break;
      case 2: batch_unit<1, true, SMALL>(P, family, unit, smem[warp]); break;
      default: batch_unit<2, true, SMALL>(P, family, unit, smem[warp]); break;
    }
    __syncwarp();                                // the staging area goes to the next unit
  }
}

// One drop-in m_kern_max (type 1) / m_kern_min (type 2) call: output blocks with explicit
// offsets, accumulated in place in the layouts mat_mult passes (type 1 reads the local
// transpose a(n3 + nd3*n1); type 2 accumulates into it).  One warp per output block.
__global__ void __launch_bounds__(256) k_dropin(int type, const int64_t* __restrict__ out_off, const int* __restrict__ dims,
                                                const int64_t* __restrict__ ptr, const int64_t* __restrict__ pairs, int n_out,
                                                const double* __restrict__ x, const double* __restrict__ b,
                                                double* __restrict__ out) {
  int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (q >= n_out) return;
  const int r = dims[2 * q], cols = dims[2 * q + 1], ne = r * cols;
  double* O = out + out_off[q];
  for (int e = lane; e < ne; e += 32) {
    double acc = O[e];
    if (type == 1) {
      int n1 = e % r, n2 = e / r;
      for (int64_t t = ptr[q]; t < ptr[q + 1]; ++t) {
        const double* X = x + pairs[3 * t];
        const double* B = b + pairs[3 * t + 1];
        int nd3 = (int)pairs[3 * t + 2];
        for (int n3 = 0; n3 < nd3; ++n3) acc = madd<true>(acc, X[n3 + nd3 * n1], B[n3 + nd3 * n2]);
      }
    } else {
      int n3 = e % cols, n1 = e / cols;   // atrans block: nd3 x nd1, n3 fastest
      for (int64_t t = ptr[q]; t < ptr[q + 1]; ++t) {
        const double* X = x + pairs[3 * t];
        const double* B = b + pairs[3 * t + 1];
        int nd2 = (int)pairs[3 * t + 2];
        for (int n2 = 0; n2 < nd2; ++n2) acc = madd<true>(acc, X[n1 + r * n2], B[n3 + cols * n2]);
      }
    }
    O[e] = acc;
  }
}

}  // namespace

void launch_dropin(int type, const int64_t* d_out, const int* d_dims, const int64_t* d_ptr, const int64_t* d_pairs,
                   int n_out, const double* x, const double* b, double* out, cudaStream_t st) {
  if (n_out <= 0) return;
  int grid = (int)(((int64_t)n_out * 32 + 255) / 256);
  k_dropin<<<grid, 256, 0, st>>>(type, d_out, d_dims, d_ptr, d_pairs, n_out, x, b, out);
  CQ_CUDA(cudaGetLastError());
}

// Output blocks by descending pair count (blocks of more than four rows first in systems of several sizes):
// the lanes of a warp get lists of similar length and the long ones start first.  A stable counting sort on the
// device (blocks of equal count keep their order: neighbours in a row share operand blocks in the caches).
namespace {
constexpr int kOrderTile = 1024;      // blocks counted and placed by one CTA

struct OrderKey {
  const int64_t* ptr;
  const int *o_row, *prim_nsf;
  int by_rows, counts;                // counts: bins per row class
  __device__ __forceinline__ int operator()(int q) const {
    const int c = (int)min(ptr[q + 1] - ptr[q], (int64_t)(counts - 1));
    return (by_rows && prim_nsf[o_row[q]] <= 4 ? counts : 0) + counts - 1 - c;
  }
};
// hist[bin * tiles + tile]: blocks of the tile in the bin
__global__ void __launch_bounds__(256) k_order_count(OrderKey key, int n, int bins, int* __restrict__ hist) {
  extern __shared__ int order_bins[];
  for (int b = threadIdx.x; b < bins; b += 256) order_bins[b] = 0;
  __syncthreads();
  for (int q = blockIdx.x * kOrderTile + threadIdx.x; q < min(n, (int)(blockIdx.x + 1) * kOrderTile); q += 256)
    atomicAdd(order_bins + key(q), 1);
  __syncthreads();
  for (int b = threadIdx.x; b < bins; b += 256) hist[(size_t)b * gridDim.x + blockIdx.x] = order_bins[b];
}
// first: the exclusive scan of hist.  The warps of a CTA place their 32 blocks one after the other.
__global__ void __launch_bounds__(256) k_order_fill(OrderKey key, int n, int bins, const int64_t* __restrict__ first,
                                                    int* __restrict__ order) {
  extern __shared__ int order_bins[];
  for (int b = threadIdx.x; b < bins; b += 256) order_bins[b] = (int)first[(size_t)b * gridDim.x + blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int q0 = blockIdx.x * kOrderTile; q0 < min(n, (int)(blockIdx.x + 1) * kOrderTile); q0 += 256) {
    const int q = q0 + threadIdx.x, bin = q < n ? key(q) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, bin);
    const int lead = __ffs(peers) - 1;
    for (int w = 0; w < 8; ++w) {
      __syncthreads();
      if (w != warp) continue;
      int at = 0;
      if (bin >= 0 && lane == lead) { at = order_bins[bin]; order_bins[bin] = at + __popc(peers); }
      at = __shfl_sync(0xffffffffu, at, lead);
      if (bin >= 0) order[at + __popc(peers & ((1u << lane) - 1u))] = q;
    }
  }
}
}  // namespace

bool capturing(const System& S) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  CQ_CUDA(cudaStreamIsCapturing(S.stream, &status));
  return status != cudaStreamCaptureStatusNone;
}

// The plan's output order, built on its first use, which allocates: null for a launch that is being captured into a graph
// before then.
static const int* output_order(System& S, ProductPlan& P) {
  const RangeIndex& O = *S.ranges[P.out_range];
  if (P.order.n != 0 || O.nnz == 0 || capturing(S)) return P.order.p;
  OrderKey key;
  key.ptr = P.ptr.p;
  key.o_row = O.nb_row.p;
  key.prim_nsf = S.dg.prim_nsf.p;
  key.by_rows = S.uniform_nsf == 0;
  // a pair list is no longer than a row of either operand; counts above 4095 share a bin
  const int longest = std::min(S.ranges[P.mult_type == 1 ? P.ra : P.rc]->max_row, S.ranges[P.rb]->max_row);
  key.counts = std::min(longest, 4095) + 1;
  const int bins = key.counts * (key.by_rows ? 2 : 1), tiles = (O.nnz + kOrderTile - 1) / kOrderTile;
  DevBuf<int> hist;
  DevBuf<int64_t> first;
  hist.alloc((size_t)bins * tiles, S.stream);
  first.alloc((size_t)bins * tiles + 1, S.stream);
  k_order_count<<<tiles, 256, bins * sizeof(int), S.stream>>>(key, O.nnz, bins, hist.p);
  CQ_CUDA(cudaGetLastError());
  dev_exclusive_scan(hist.p, (int64_t)bins * tiles, first.p, S.stream);   // nothing here waits for the device
  P.order.alloc(O.nnz, S.stream);
  k_order_fill<<<tiles, 256, bins * sizeof(int), S.stream>>>(key, O.nnz, bins, first.p, P.order.p);
  S.launches += 2;
  CQ_CUDA(cudaGetLastError());
  return P.order.p;
}

// Dynamic shared memory above 48 KB has to be allowed per kernel (once per system and kernel).
template <class K>
static void allow_smem(System& S, K* kern, int bytes) {
  const void* k = reinterpret_cast<const void*>(kern);
  if (!S.smem_allowed.insert(k).second) return;
  CQ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

// The generic kernel, which needs no output order: 32 R elements per block.
static void launch_generic(const System& S, const ProductPlan& P, const MultArgs& M, int exact, cudaStream_t st) {
  const int T = 256, grid = (int)(((int64_t)M.n_out * 32 + T - 1) / T);
  auto by_type = [&](auto r) {
    constexpr int R = decltype(r)::value;
    if (P.mult_type == 1) {
      if (exact) k_mult_generic<1, true, R><<<grid, T, 0, st>>>(M, S.uniform_nsf);
      else k_mult_generic<1, false, R><<<grid, T, 0, st>>>(M, S.uniform_nsf);
    } else {
      if (exact) k_mult_generic<2, true, R><<<grid, T, 0, st>>>(M, S.uniform_nsf);
      else k_mult_generic<2, false, R><<<grid, T, 0, st>>>(M, S.uniform_nsf);
    }
  };
  if (S.max_nsf <= 5) by_type(std::integral_constant<int, 1>{});
  else if (S.max_nsf <= 8) by_type(std::integral_constant<int, 2>{});
  else by_type(std::integral_constant<int, 8>{});
  CQ_CUDA(cudaGetLastError());
}

// One launch of the FP64 product with kernel `variant` (0..6 for uniform 4 x 4 blocks with 16-byte aligned operands; for
// anything else 4 is the group kernel and every other number the generic one).  All variants give the same
// bits: they differ only in how the work is mapped onto the GPU.
static void launch_variant(System& S, ProductPlan& P, const MultArgs& M, int variant, int exact, bool nd4) {
  cudaStream_t st = S.stream;
  const int T = 256;
  RangeIndex& O = P.mult_type == 1 ? *S.ranges[P.rc] : *S.ranges[P.ra];
  RangeIndex& X = P.mult_type == 1 ? *S.ranges[P.ra] : *S.ranges[P.rc];
  // the row kernel's tiles are uploaded on its first use: a launch captured before then takes another kernel
  if (nd4 && variant == 4 && P.mult_type == 2 && P.n_row_tiles < 0 && capturing(S)) variant = 3;
  const bool row_kernel = nd4 && variant == 4 && P.mult_type == 2;        // the row kernel has an order of its own
  // the staged kernels take their output order without a test for its absence (the test alone cost the smallest products
  // 2 to 4 %): a launch captured before the order exists runs variant 0, which has none
  const int* order = nullptr;
  if ((nd4 ? variant >= 3 && !row_kernel : variant == 4) && !(order = output_order(S, P))) variant = 0;
  if (nd4 && variant == 6) {
    const int grid = (M.n_out + 127) / 128;
    const size_t smem = (size_t)4 * kBulkStages * 64 * kBulkSlot;
    int* err = device_timeout_word(S);
    auto launch = [&](auto kern) {
      allow_smem(S, kern, (int)smem);
      kern<<<grid, 128, smem, st>>>(M, order, err);
    };
    if (P.mult_type == 1) {
      if (exact) launch(k_mult_nd4_bulk<1, true>); else launch(k_mult_nd4_bulk<1, false>);
    } else {
      if (exact) launch(k_mult_nd4_bulk<2, true>); else launch(k_mult_nd4_bulk<2, false>);
    }
  } else if (nd4 && variant == 5) {
    const int grid = (M.n_out + 31) / 32;        // 8 output blocks per warp, 4 warps per CTA
    if (P.mult_type == 1) {
      if (exact) k_mult_nd4_quad<1, true, 4><<<grid, 128, 0, st>>>(M, order);
      else k_mult_nd4_quad<1, false, 4><<<grid, 128, 0, st>>>(M, order);
    } else {
      if (exact) k_mult_nd4_quad<2, true, 4><<<grid, 128, 0, st>>>(M, order);
      else k_mult_nd4_quad<2, false, 4><<<grid, 128, 0, st>>>(M, order);
    }
  } else if (row_kernel) {
    if (P.n_row_tiles < 0) {
      // up to 32 output blocks whose column atoms are images of one atom, with that atom's row of B
      RangeIndex& B = *S.ranges[P.rb];
      std::vector<int4> tl;
      for (int k = 0; k < S.geo.n_prim; ++k)
        for (int z = O.h_row_ptr[k]; z < O.h_row_ptr[k + 1]; z += 32)
          tl.push_back(make_int4(B.h_row_ptr[k], B.h_row_ptr[k + 1], z, std::min(32, O.h_row_ptr[k + 1] - z)));
      P.row_tiles.upload(tl, st);
      P.n_row_tiles = (int)tl.size();
    }
    constexpr int kSt = 2;
    const int smem = 2 * kSt * (4096 + 128), grid = (P.n_row_tiles + 1) / 2;
    if (exact) k_mult_nd4_row<true, kSt><<<grid, 64, smem, st>>>(M, P.row_tiles.p, P.n_row_tiles, O.trans_dest.p);
    else k_mult_nd4_row<false, kSt><<<grid, 64, smem, st>>>(M, P.row_tiles.p, P.n_row_tiles, O.trans_dest.p);
  } else if (nd4 && (variant == 3 || variant == 4)) {
    const int grid = (M.n_out + 127) / 128;
    if (P.mult_type == 1) {
      if (exact) k_mult_nd4_warp<1, true><<<grid, 128, 0, st>>>(M, order);
      else k_mult_nd4_warp<1, false><<<grid, 128, 0, st>>>(M, order);
    } else {
      if (exact) k_mult_nd4_warp<2, true><<<grid, 128, 0, st>>>(M, order);
      else k_mult_nd4_warp<2, false><<<grid, 128, 0, st>>>(M, order);
    }
  } else if (nd4 && variant == 2) {
    constexpr int kChunk = 256;                 // 32 KiB of operand blocks per chunk
    if (P.n_tiles == 0) {
      // tiles: up to 128 output blocks of one row, with that row's range of operand blocks
      std::vector<int4> tl;
      for (int i = 0; i < S.geo.n_prim; ++i)
        for (int q0 = O.h_row_ptr[i]; q0 < O.h_row_ptr[i + 1]; q0 += 128)
          tl.push_back(make_int4(q0, std::min(q0 + 128, O.h_row_ptr[i + 1]), X.h_row_ptr[i], X.h_row_ptr[i + 1]));
      P.tiles.upload(tl, st);
      P.n_tiles = (int)tl.size();
    }
    if (P.mult_type == 1) {
      if (exact) k_mult_nd4_rows<1, true, kChunk><<<P.n_tiles, 128, 0, st>>>(M, P.tiles.p);
      else k_mult_nd4_rows<1, false, kChunk><<<P.n_tiles, 128, 0, st>>>(M, P.tiles.p);
    } else {
      if (exact) k_mult_nd4_rows<2, true, kChunk><<<P.n_tiles, 128, 0, st>>>(M, P.tiles.p);
      else k_mult_nd4_rows<2, false, kChunk><<<P.n_tiles, 128, 0, st>>>(M, P.tiles.p);
    }
  } else if (nd4 && variant == 1) {
    const int T1 = 128;
    int grid = (M.n_out + T1 - 1) / T1;
    if (P.mult_type == 1) {
      if (exact) k_mult_nd4_tpb<1, true><<<grid, T1, 0, st>>>(M); else k_mult_nd4_tpb<1, false><<<grid, T1, 0, st>>>(M);
    } else {
      if (exact) k_mult_nd4_tpb<2, true><<<grid, T1, 0, st>>>(M); else k_mult_nd4_tpb<2, false><<<grid, T1, 0, st>>>(M);
    }
  } else if (nd4) {
    int grid = (int)(((int64_t)M.n_out * 16 + T - 1) / T);
    if (P.mult_type == 1) {
      if (exact) k_mult_nd4<1, true><<<grid, T, 0, st>>>(M); else k_mult_nd4<1, false><<<grid, T, 0, st>>>(M);
    } else {
      if (exact) k_mult_nd4<2, true><<<grid, T, 0, st>>>(M); else k_mult_nd4<2, false><<<grid, T, 0, st>>>(M);
    }
  } else if (variant == 4) {
    auto launch = [&](auto kern, int blocks, int warp_bytes) {
      kern<<<(M.n_out + 2 * blocks - 1) / (2 * blocks), 64, 2 * warp_bytes, st>>>(M, order);
    };
    auto by_size = [&](auto type, auto ex) {
      constexpr int TY = decltype(type)::value;
      constexpr bool EX = decltype(ex)::value;
      auto by_group = [&](auto lpb, auto stages) {
        constexpr int LPB = decltype(lpb)::value, ST = decltype(stages)::value;
        if (S.uniform_nsf == 13) launch(k_mult_group<TY, EX, 13, 13, LPB, ST>, 32 / LPB, GroupShape<13, LPB, ST>::kWarpBytes);
        else if (S.max_nsf <= 13) launch(k_mult_group<TY, EX, 0, 13, LPB, ST>, 32 / LPB, GroupShape<13, LPB, ST>::kWarpBytes);
        else launch(k_mult_group<TY, EX, 0, 16, LPB, ST>, 32 / LPB, GroupShape<16, LPB, ST>::kWarpBytes);
      };
      // four blocks per warp once they give every SM its 18 resident warps: past the 8,000 output blocks where the two
      // shapes are equal (see k_mult_group)
      if (M.n_out >= 148 * 18 * 4) by_group(std::integral_constant<int, 8>{}, std::integral_constant<int, 1>{});
      else by_group(std::integral_constant<int, 16>{}, std::integral_constant<int, 2>{});
    };
    using std::integral_constant;
    if (P.mult_type == 1) {
      if (exact) by_size(integral_constant<int, 1>{}, std::true_type{}); else by_size(integral_constant<int, 1>{}, std::false_type{});
    } else {
      if (exact) by_size(integral_constant<int, 2>{}, std::true_type{}); else by_size(integral_constant<int, 2>{}, std::false_type{});
    }
  } else {
    launch_generic(S, P, M, exact, st);
  }
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}

// Kernel of an FP64 product when none is forced: a rule on the product's sizes (every kernel gives the same bits).
// Timing the candidates on a product's first call, as this library once did, cost a new geometry several times
// the product and chose wrongly while other streams kept the device busy.  Measured on cells of 64 to 1000 atoms
// and ranges of 8 to 26 bohr (warp-staged / four lanes per block / row kernel, us):
//  - type 1: four lanes per block below 180,000 output blocks (7940: 12.9 / 7.9; 85,546: 37.5 / 22.9; 163,036: 27.1 /
//    27.0; 217,306: 31.2 / 33.2; 1,182,142: 580 / 716);
//  - type 2: four lanes per block below 20,000 output blocks (7940 with 532 pairs each: 302 / 148 / 234; 18,048: 465 /
//    248 / 316; 24,064: 472 / 378 / 322); above, the row kernel, whose steps are the rows of B: where the lists
//    hold most of those rows, and from 40,000 blocks on (every SM full) also most lanes have a block (63,664 with
//    97 % of the lanes: 605 / 823 / 570; 47,000 with 73 %: 520 / 625 / 611; lists of 88 %: 127 / 170 / 135).
// Other block sizes and unaligned operands: the group kernel (on 13 x 13 blocks the generic one is 2 to 3 times slower),
// except for small blocks in few output blocks, whose time is the latency of a step and not its arithmetic (generic /
// group, us): blocks of up to 5 rows below 17,000 output blocks (1600 of 1 and 4 rows 11.9 / 22.5; 6298 55.6 / 86.2; 15,342
// equal; 71,030 67.3 / 60.9), of 6 to 8 below 2,000 (1862 of 8 x 8 43.6 / 60.2; 3016 86 / 100 in the group's favour).
static int auto_variant(System& S, ProductPlan& P, int n_out, bool nd4) {
  if (!nd4) {
    const int variant = n_out < (S.max_nsf <= 5 ? 17000 : S.max_nsf <= 8 ? 2000 : 0) ? 0 : 4;
    if (S.uniform_nsf != 4) P.tuned = variant;
    return variant;
  }
  if (P.tuned >= 0) return P.tuned;
  if (P.mult_type == 1) return P.tuned = n_out < 180000 ? 5 : 3;
  if (n_out < 20000) return P.tuned = 5;
  const std::vector<int>&o = S.ranges[P.ra]->h_row_ptr, &b = S.ranges[P.rb]->h_row_ptr;
  int64_t steps = 0, tiles = 0;                  // pairs if every list held its whole row of B; groups of 32 blocks
  for (int k = 0; k < S.geo.n_prim; ++k) {
    steps += (int64_t)(o[k + 1] - o[k]) * (b[k + 1] - b[k]);
    tiles += (o[k + 1] - o[k] + 31) / 32;
  }
  const double lists = (double)P.n_pairs / (double)std::max<int64_t>(steps, 1), lanes = n_out / (32.0 * (double)tiles);
  return P.tuned = n_out < 40000 ? (lists >= 0.75 ? 4 : 3) : (lists >= 0.9 && lanes >= 0.8 ? 4 : 3);
}

// FP64 tensor-core products whose time is latency: the short-list kernel, without an output order.  Not for one block size
// of 13 (compiled in) or sizes up to 8 (one MMA tile per block), where the staged kernel is the faster one at every size.
// Measured (staged / short, us): 4 and 13 rows, 3008 output blocks of 0.5 terms 6.0 / 5.5, 1600 of 12 19.1 / 16.0, 8070 of
// 3.8 14.8 / 19.2, 2078 of 28 24.7 / 27.1; 5 and 13 rows, 2078 of 0.7 6.3 / 4.7, 4530 of 4.0 15.1 / 14.2, 10,100 of 3.1
// 18.1 / 23.6; 16 x 16 blocks, 1600 of 12 37.5 / 23.8, 6288 of 9.3 51.5 / 47.5, 12,900 of 8.1 77.8 / 76.7, 3406 of 31 67.2 / 77.9.
static bool dmma_short(const System& S, const ProductPlan& P, int n_out) {
  if (S.uniform_nsf == 13 || S.max_nsf <= 8) return false;
  return S.max_nsf <= 13 ? n_out < 5000 && P.n_pairs < 50000 : P.n_pairs < 100000;
}

// kernel arguments of one product (roles of mat_mult: type 1 writes c from a, b; type 2 writes a from c, b);
// nd4: uniform 4 x 4 blocks with 16-byte aligned operands (the 4 x 4 kernels read 16-byte vectors)
static MultArgs product_args(System& S, ProductPlan& P, double* a, const double* b, double* c, bool* nd4) {
  RangeIndex &A = *S.ranges[P.ra], &B = *S.ranges[P.rb], &C = *S.ranges[P.rc];
  MultArgs M;
  M.ptr = P.ptr.p;
  M.pairs = P.pairs.p;
  M.b_elem = B.nb_elem.p;
  M.b_cover = B.nb_cover.p;
  M.prim_nsf = S.dg.prim_nsf.p;
  M.cover_nsf = S.dg.cover_nsf.p;
  M.b = b;
  RangeIndex& O = P.mult_type == 1 ? C : A;
  RangeIndex& X = P.mult_type == 1 ? A : C;
  M.n_out = O.nnz;
  M.o_row = O.nb_row.p; M.o_cover = O.nb_cover.p; M.o_elem = O.nb_elem.p;
  M.x_cover = X.nb_cover.p; M.x_elem = X.nb_elem.p;
  M.x = P.mult_type == 1 ? a : c;
  M.out = P.mult_type == 1 ? c : a;
  const bool aligned = ((uintptr_t)b % 16 == 0) && ((uintptr_t)M.x % 16 == 0) && ((uintptr_t)M.out % 16 == 0);
  *nd4 = S.uniform_nsf == 4 && aligned;
  return M;
}

void launch_mat_mult(System& S, ProductPlan& P, double* a, const double* b, double* c, int exact) {
  RangeIndex &A = *S.ranges[P.ra], &B = *S.ranges[P.rb], &C = *S.ranges[P.rc];
  bool nd4 = false;
  MultArgs M = product_args(S, P, a, b, c, &nd4);
  if (M.n_out == 0) return;
  cudaStream_t st = S.stream;
  cudaEvent_t ev0 = nullptr;
  if (S.prof.on) { ev0 = S.prof.get(); CQ_CUDA(cudaEventRecord(ev0, st)); }
  // fused multiply-add products of blocks larger than 8 x 8 run on the FP64 tensor cores: an m8n8k4 MMA
  // chains its four products into the accumulator as fused multiply-adds in k order, so the bits are
  // those of the CUDA-core kernels (checked on B200; unless a CUDA-core variant is forced with CQ_OPT_MULT_VARIANT).
  // Tensor cores / group kernel with fused multiply-add, us: LS.L -> LSL of 64 DZP atoms 1396 / 1639, LS.S -> SLS of 216
  // 1223 / 1409, 216 atoms 8, 12 -> 20 bohr 84 / 86, 16 x 16 blocks 176 / 236, 5 and 13 rows 267 / 324, 9 x 9 267 / 270,
  // 4 and 13 rows 235 / 214 (type 1) and 180 / 202 (type 2), 656 output blocks of a cluster 12.5 / 26.7
  if (exact == kPrecFp64Tensor || (exact == 0 && S.max_nsf > 8 && S.mult_variant == kVariantAuto)) {
    if (dmma_short(S, P, M.n_out)) {
      const int grid = (M.n_out + 3) / 4;
      if (P.mult_type == 1) k_mult_dmma_short<1><<<grid, 128, 0, st>>>(M);
      else k_mult_dmma_short<2><<<grid, 128, 0, st>>>(M);
    } else {
      // below 1,200 output blocks every SM holds its share at once: the order would cost a first call more than it gives
      const int* order = M.n_out < 1200 ? nullptr : output_order(S, P);
      const int grid = (M.n_out + 1) / 2;
      if (P.mult_type == 1) {
        if (S.uniform_nsf == 13) k_mult_dmma<1, 13, 13><<<grid, 64, 0, st>>>(M, order);
        else if (S.max_nsf <= 13) k_mult_dmma<1, 0, 13><<<grid, 64, 0, st>>>(M, order);
        else k_mult_dmma<1, 0, 16><<<grid, 64, 0, st>>>(M, order);
      } else {
        if (S.uniform_nsf == 13) k_mult_dmma<2, 13, 13><<<grid, 64, 0, st>>>(M, order);
        else if (S.max_nsf <= 13) k_mult_dmma<2, 0, 13><<<grid, 64, 0, st>>>(M, order);
        else k_mult_dmma<2, 0, 16><<<grid, 64, 0, st>>>(M, order);
      }
    }
    S.launches++;
    CQ_CUDA(cudaGetLastError());
  } else {
    int variant = S.mult_variant;
    if (variant == kVariantAuto) variant = auto_variant(S, P, M.n_out, nd4);
    launch_variant(S, P, M, variant, exact, nd4);
  }
  if (S.prof.on) {
    cudaEvent_t ev1 = S.prof.get();
    CQ_CUDA(cudaEventRecord(ev1, st));
    // algorithmic bytes: read both operands once, write the result once (8 bytes per element)
    double bytes = 8.0 * (double)(A.length + B.length + C.length);
    S.prof.recs.push_back({ev0, ev1, bytes, (double)P.flops});
  }
}

void ensure_product_order(System& S, ProductPlan& P) { output_order(S, P); }

// A batch whose products are all of small blocks (other than aligned 4 x 4) runs the generic kernel, in the stored order.
// Six products of a system, us, group / generic: 60 atoms of 1 and 4 rows (3548 and 1014 output blocks) 82.8 / 54.8, of 5 x 5
// 107.9 / 55.3, 150 atoms of 1 x 1 (4432, 624) 17.5 / 10.9; but 16,676 and 3016 of 1 x 1 119.7 / 132.2.  One kernel per call:
// next to the other bodies the generic one made the registers of all spill (every other product a third slower), and two
// launches in a row lose what their overlap gives.
bool batch_of_small_blocks(const std::vector<BatchItem>& items) {
  for (const BatchItem& it : items)
    if (it.S->uniform_nsf == 4 || it.S->max_nsf > 5 || it.S->ranges[it.P->out_range]->nnz >= 10000) return false;
  return true;
}

// Products of independent systems (or of one system) in persistent launches on `st` (up to kBatchMax
// products each).  The caller orders `st` after the work the operands depend on and the systems' later
// work after it.
void launch_mat_mult_batch(const std::vector<BatchItem>& items, cudaStream_t st) {
  int dev_id = 0, sms = 0, occ = 0;
  CQ_CUDA(cudaGetDevice(&dev_id));
  CQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_id));
  const bool small = batch_of_small_blocks(items);
  auto params = std::make_unique<BatchParams>();
  BatchParams& B = *params;
  auto flush = [&] {
    if (B.n_prod == 0) return;
    const int n_units = B.unit_off[B.n_prod];
    auto* kern = small ? k_mult_batch<true> : k_mult_batch<false>;
    CQ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 128, 0));
    const int grid = std::max(1, std::min(sms * std::max(occ, 1), (n_units + 3) / 4));
    kern<<<grid, 128, 0, st>>>(B);
    CQ_CUDA(cudaGetLastError());
    B.n_prod = 0;
  };
  B.n_prod = 0;
  B.unit_off[0] = 0;
  for (const BatchItem& it : items) {
    System& S = *it.S;
    ProductPlan& P = *it.P;
    bool nd4 = false;
    BatchProduct bp;
    bp.M = product_args(S, P, it.a, it.b, it.c, &nd4);
    if (bp.M.n_out == 0) continue;
    bp.order = P.order.p;              // built by ensure_product_order on the system's stream
    if (!small && !bp.order) {         // captured before it exists: a launch of its own
      launch_generic(S, P, bp.M, it.exact, st);
      S.launches++;
      continue;
    }
    bp.kind = (P.mult_type == 2 ? 1 : 0) | (it.exact ? 2 : 0) |
              (nd4 ? kBatchNd4 : S.uniform_nsf == 13 ? kBatchU13 : S.max_nsf <= 13 ? kBatchMax13 : kBatchMax16);
    bp.u = S.uniform_nsf;
    if (B.n_prod == kBatchMax) { flush(); B.unit_off[0] = 0; }
    B.prods[B.n_prod] = bp;
    const int per_unit = small ? 1 : nd4 ? 32 : 2;
    B.unit_off[B.n_prod + 1] = B.unit_off[B.n_prod] + (bp.M.n_out + per_unit - 1) / per_unit;
    ++B.n_prod;
    S.launches++;
  }
  flush();
}

cudaEvent_t ProductProfile::get() {
  if (!spare.empty()) { cudaEvent_t e = spare.back(); spare.pop_back(); return e; }
  cudaEvent_t e;
  CQ_CUDA(cudaEventCreate(&e));
  return e;
}
void ProductProfile::clear() {
  for (auto& r : recs) { spare.push_back(r.a); spare.push_back(r.b); }
  recs.clear();
}
ProductProfile::~ProductProfile() {
  clear();
  for (cudaEvent_t e : spare) cudaEventDestroy(e);
}

}  // namespace cqb
