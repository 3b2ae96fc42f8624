// Split-precision block products on the tensor cores (blocks of up to 16 x 16).
//
// Each FP64 operand block is padded to 16 x 16 and split into two bf16 parts,
// v = hi + lo (hi = bf16(v), lo = bf16(v - hi)); a block product is the sum of
// hi.hi + hi.lo + lo.hi (three bf16 MMAs, FP32 accumulation), which carries
// about 16 significant bits per term.  The three-part split (v = hi + mid + lo,
// six MMAs per term, FP64 accumulation across terms) carries about 22.  The result is written back as FP64 into
// the block storage of the output range, so the matrices of the chain stay FP64.
//
// Work decomposition (output stationary): one warp owns one output block and takes the terms of its pair list,
// sorted by the first operand block (A_ik for type 1, C_ij for type 2), in order.  Operands are pre-converted
// into the per-lane fragment order of mma.m16n8k16, so every fragment is one coalesced 16-byte load per lane.
#include <cuda_bf16.h>

#include <algorithm>

#include "cq_internal.hpp"


namespace cqb {
namespace {


__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo_k, __nv_bfloat16 hi_k) {
  return (uint32_t)__bfloat16_as_ushort(lo_k) | ((uint32_t)__bfloat16_as_ushort(hi_k) << 16);
}

// element (r, c) of a padded 16 x 16 view of a column-major nd_r x nd_c FP64 block
__device__ __forceinline__ double blk_at(const double* B, int nd_r, int nd_c, int r, int c) {
  return (r < nd_r && c < nd_c) ? B[r + nd_r * c] : 0.0;
}

__device__ __forceinline__ void split2(double v, __nv_bfloat16& h, __nv_bfloat16& l) {
  h = __double2bfloat16(v);
  l = __double2bfloat16(v - (double)__bfloat162float(h));
}

// v = hi + mid + lo + r with |r| <= 2^-24 |v| (about 2^-25 for round-to-nearest parts): both
// differences are exact in FP64
__device__ __forceinline__ void split3(double v, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
  h = __double2bfloat16(v);
  const double r1 = v - (double)__bfloat162float(h);
  m = __double2bfloat16(r1);
  l = __double2bfloat16(r1 - (double)__bfloat162float(m));
}

// A-role fragments (M = block rows, K = block columns):
//   reg0 (row g,   k 2t..2t+1), reg1 (row g+8, k 2t..2t+1), reg2 (row g, k 2t+8..), reg3 (row g+8, k 2t+8..)
// B-role fragments (K = block rows, N = block columns; `trans` uses the transposed block),
//   two n8 tiles: {tile0 (k 2t.., n g), tile0 (k 2t+8.., n g), tile1 (k 2t.., n g+8), tile1 (k 2t+8.., n g+8)}
__global__ void k_to_frag(int nnz, const int64_t* __restrict__ elem, const int* __restrict__ row,
                          const int* __restrict__ cover, const int* __restrict__ prim_nsf,
                          const int* __restrict__ cover_nsf, const double* __restrict__ src, int role_b, int trans,
                          uint4* __restrict__ hi, uint4* __restrict__ lo, uint4* __restrict__ mid) {
  int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int e = (int)(tid >> 5), lane = (int)(tid & 31);
  if (e >= nnz) return;
  const int ndr = prim_nsf[row[e]], ndc = cover_nsf[cover[e]];
  const double* B = src + elem[e];
  const int g = lane >> 2, t = lane & 3;
  int rr[8], cc[8];
  if (!role_b) {
    const int r0[4] = {g, g + 8, g, g + 8}, c0[4] = {2 * t, 2 * t, 2 * t + 8, 2 * t + 8};
    for (int q = 0; q < 4; ++q) { rr[2 * q] = r0[q]; cc[2 * q] = c0[q]; rr[2 * q + 1] = r0[q]; cc[2 * q + 1] = c0[q] + 1; }
  } else {
    // (K, N) pairs; element (K=k, N=n) is block (k, n), or block (n, k) when transposed
    const int k0[4] = {2 * t, 2 * t + 8, 2 * t, 2 * t + 8}, n0[4] = {g, g, g + 8, g + 8};
    for (int q = 0; q < 4; ++q) {
      for (int h = 0; h < 2; ++h) {
        int k = k0[q] + h, n = n0[q];
        rr[2 * q + h] = trans ? n : k;
        cc[2 * q + h] = trans ? k : n;
      }
    }
  }
  uint32_t wh[4], wm[4], wl[4];
  for (int q = 0; q < 4; ++q) {
    __nv_bfloat16 h0, m0, l0, h1, m1, l1;
    const double v0 = blk_at(B, ndr, ndc, rr[2 * q], cc[2 * q]), v1 = blk_at(B, ndr, ndc, rr[2 * q + 1], cc[2 * q + 1]);
    if (mid) {
      split3(v0, h0, m0, l0);
      split3(v1, h1, m1, l1);
      wm[q] = pack_bf16(m0, m1);
    } else {
      split2(v0, h0, l0);
      split2(v1, h1, l1);
    }
    wh[q] = pack_bf16(h0, h1);
    wl[q] = pack_bf16(l0, l1);
  }
  hi[(int64_t)e * 32 + lane] = make_uint4(wh[0], wh[1], wh[2], wh[3]);
  lo[(int64_t)e * 32 + lane] = make_uint4(wl[0], wl[1], wl[2], wl[3]);
  if (mid) mid[(int64_t)e * 32 + lane] = make_uint4(wm[0], wm[1], wm[2], wm[3]);
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

struct TCArgs {
  int n_out;
  const int64_t* __restrict__ ptr;     // pair list offsets per output block
  const int2* __restrict__ pairs;      // (first-operand block, B block), first operand ascending
  const uint4* __restrict__ xa_hi;     // first operand, A-role fragments
  const uint4* __restrict__ xa_lo;
  const uint4* __restrict__ bb_hi;     // B operand, B-role fragments
  const uint4* __restrict__ bb_lo;
  const uint4* __restrict__ xa_mid;    // middle parts (three-part split only)
  const uint4* __restrict__ bb_mid;
  const int* __restrict__ o_row;
  const int* __restrict__ o_cover;
  const int64_t* __restrict__ o_elem;
  const int* __restrict__ prim_nsf;
  const int* __restrict__ cover_nsf;
  double* __restrict__ out;
};

// the accumulators (rows g and g + 8, columns 2 t4 and 2 t4 + 1 of each n8 half) to output block q
template <class Acc>
__device__ __forceinline__ void store_block(const TCArgs& M, int q, int lane, const Acc (&acc)[2][4]) {
  const int g = lane >> 2, t4 = lane & 3;
  const int ndr = M.prim_nsf[M.o_row[q]], ndc = M.cover_nsf[M.o_cover[q]];
  double* O = M.out + M.o_elem[q];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      int row = g + ((r & 2) ? 8 : 0), col = 8 * h + 2 * t4 + (r & 1);
      if (row < ndr && col < ndc) O[row + ndr * col] = (double)acc[h][r];
    }
}

// Two-part split (BF16x3), one output block per warp: three MMAs per pair and n8 half into FP32 accumulators, the
// halves alternating so that neither chain waits for its own last MMA.  The next term's fragments are loaded
// while the current term's MMAs run, and the pair after that a term earlier still, so that no load waits for
// another.  What bounds it: the 2 KB of fragments a pair brings from L2 (32 cycles at 64 bytes per SM and cycle; it
// takes 32 on LS.L -> LSL of the 216-atom DZP cell, 40.3 TFLOP/s; without the alternation and the early pair 38.8).
// Not taken: groups of 2, 4 and 8 output blocks of a row that share first-operand fragments (1744, 2290 and 4118 us
// against 1620 there: the union of their lists is longer than what they share); copies into shared memory with
// cp.async (1732 us); 8-byte loads that skip the padding rows (2154 us: twice the requests).
__global__ void __launch_bounds__(128) k_mult_split2(TCArgs M) {
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (q >= M.n_out) return;
  const int2* pairs = M.pairs + M.ptr[q];
  const int nt = (int)(M.ptr[q + 1] - M.ptr[q]);
  float acc[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[h][r] = 0.f;
  struct Term { uint4 ah, al, bh, bl; };
  auto load = [&](int2 pr) {
    Term v;
    v.ah = __ldg(M.xa_hi + (int64_t)pr.x * 32 + lane);
    v.al = __ldg(M.xa_lo + (int64_t)pr.x * 32 + lane);
    v.bh = __ldg(M.bb_hi + (int64_t)pr.y * 32 + lane);
    v.bl = __ldg(M.bb_lo + (int64_t)pr.y * 32 + lane);
    return v;
  };
  Term cur = {}, nxt = {};
  int2 pn = make_int2(0, 0);
  if (nt > 0) cur = load(__ldg(pairs));
  if (nt > 1) pn = __ldg(pairs + 1);
  for (int t = 0; t < nt; ++t) {
    if (t + 1 < nt) nxt = load(pn);
    if (t + 2 < nt) pn = __ldg(pairs + t + 2);
    mma_bf16(acc[0], cur.al, cur.bh.x, cur.bh.y);
    mma_bf16(acc[1], cur.al, cur.bh.z, cur.bh.w);
    mma_bf16(acc[0], cur.ah, cur.bl.x, cur.bl.y);
    mma_bf16(acc[1], cur.ah, cur.bl.z, cur.bl.w);
    mma_bf16(acc[0], cur.ah, cur.bh.x, cur.bh.y);
    mma_bf16(acc[1], cur.ah, cur.bh.z, cur.bh.w);
    cur = nxt;
  }
  store_block(M, q, lane, acc);
}

__device__ __forceinline__ void lane_copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 lane_read16(uint32_t src) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(src) : "memory");
  return v;
}

// Three-part split (BF16x6): v = hi + mid + lo, one output block per warp.  Per term and n8 half the
// six products that carry terms down to 2^-16 of hi.hi run into a zeroed FP32 accumulator, smallest
// first (hi.lo, lo.hi, mid.mid, hi.mid, mid.hi, hi.hi), and the term's 16 x 8 result is added to FP64
// accumulators, so the FP32 rounding spans one 16-wide contraction rather than the whole sum.  The
// omitted products (mid.lo, lo.mid, lo.lo) and the split remainders are below 2^-23 of |a||b| per
// element product.  The halves' MMAs alternate, as above.
// The fragments of the next two terms are on their way to shared memory (cp.async past the L1): every lane copies
// exactly the 16-byte pieces that it reads back, so no lane waits for another and the ring only stands in for
// registers (62 a thread instead of 96).  What bounds it: the 3 KB a pair brings from L2 (48 cycles); it takes 61 on
// LS.L -> LSL of the 216-atom DZP cell.  Measured on the eight products of its LNV call: three stages 12.87 ms, two
// 13.03, four 13.95; fragments prefetched into registers 13.99, with groups of two blocks 15.5 (as above).
constexpr int kSplitStages = 3;
constexpr int kSplitStep = 6 * 512;                // bytes of one term: three parts of two blocks

__global__ void __launch_bounds__(128) k_mult_split3(TCArgs M) {
  __shared__ __align__(128) unsigned char smem[4][kSplitStages * kSplitStep];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = blockIdx.x * 4 + warp;
  if (q >= M.n_out) return;
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(smem[warp]) + lane * 16;
  const int2* pairs = M.pairs + M.ptr[q];
  const int nt = (int)(M.ptr[q + 1] - M.ptr[q]);
  double acc[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[h][r] = 0.0;
  int issued = 0;
  int2 pn = nt > 0 ? __ldg(pairs) : make_int2(0, 0), pn2 = nt > 1 ? __ldg(pairs + 1) : make_int2(0, 0);
  auto issue = [&](int st) {
    if (issued < nt) {
      const uint32_t d = mine + st * kSplitStep;
      const int64_t xo = (int64_t)pn.x * 32 + lane, bo = (int64_t)pn.y * 32 + lane;
      lane_copy16(d, M.xa_hi + xo);
      lane_copy16(d + 512, M.xa_mid + xo);
      lane_copy16(d + 1024, M.xa_lo + xo);
      lane_copy16(d + 1536, M.bb_hi + bo);
      lane_copy16(d + 2048, M.bb_mid + bo);
      lane_copy16(d + 2560, M.bb_lo + bo);
      pn = pn2;
      if (issued + 2 < nt) pn2 = __ldg(pairs + issued + 2);
    }
    ++issued;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int k = 0; k + 1 < kSplitStages; ++k) issue(k);
  int st = 0;
  for (int t = 0; t < nt; ++t) {
    issue(st == 0 ? kSplitStages - 1 : st - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kSplitStages - 1) : "memory");
    const uint32_t d = mine + st * kSplitStep;
    const uint4 ah = lane_read16(d), am = lane_read16(d + 512), al = lane_read16(d + 1024);
    const uint4 bh = lane_read16(d + 1536), bm = lane_read16(d + 2048), bl = lane_read16(d + 2560);
    float c[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int r = 0; r < 4; ++r) c[h][r] = 0.f;
    mma_bf16(c[0], ah, bl.x, bl.y);
    mma_bf16(c[1], ah, bl.z, bl.w);
    mma_bf16(c[0], al, bh.x, bh.y);
    mma_bf16(c[1], al, bh.z, bh.w);
    mma_bf16(c[0], am, bm.x, bm.y);
    mma_bf16(c[1], am, bm.z, bm.w);
    mma_bf16(c[0], ah, bm.x, bm.y);
    mma_bf16(c[1], ah, bm.z, bm.w);
    mma_bf16(c[0], am, bh.x, bh.y);
    mma_bf16(c[1], am, bh.z, bh.w);
    mma_bf16(c[0], ah, bh.x, bh.y);
    mma_bf16(c[1], ah, bh.z, bh.w);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[h][r] += (double)c[h][r];
    st = st + 1 == kSplitStages ? 0 : st + 1;
  }
  store_block(M, q, lane, acc);
}

}  // namespace

// A-role (first operand) or B-role fragments of a whole range, hi and lo parts (1 KB per block)
// (and the middle parts of the three-part split when `mid` is given)
void to_fragments(System& S, int r, const double* src, int role_b, int trans, uint4* hi, uint4* lo, uint4* mid) {
  RangeIndex& R = *S.ranges[r];
  if (R.nnz == 0) return;
  int64_t threads = (int64_t)R.nnz * 32;
  k_to_frag<<<(int)((threads + 255) / 256), 256, 0, S.stream>>>(R.nnz, R.nb_elem.p, R.nb_row.p, R.nb_cover.p,
                                                                S.dg.prim_nsf.p, S.dg.cover_nsf.p, src, role_b, trans,
                                                                hi, lo, mid);
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}

static FragBuf& frag_buffer(System& S, int r, int slot, bool three = false) {
  FragBuf& f = S.frags[std::make_pair(r, slot)];
  size_t need = (size_t)std::max(S.ranges[r]->nnz, 1) * 32;
  if (f.hi.n < need) { f.hi.alloc(need, S.stream); f.lo.alloc(need, S.stream); }
  if (three && f.mid.n < need) f.mid.alloc(need, S.stream);
  return f;
}

// split-precision products on mma.sync, one output block per warp
static void mat_mult_mma_sync(System& S, MixedPlan& MP, int mult_type, int ra, int rb, int rc, double* a,
                              const double* b, double* c, int parts) {
  const int rx = mult_type == 1 ? ra : rc;
  const double* x = mult_type == 1 ? a : c;
  double* out = mult_type == 1 ? c : a;
  const bool three = parts == 3;
  FragBuf& fx = frag_buffer(S, rx, 0, three);
  FragBuf& fb = frag_buffer(S, rb, 1, three);
  to_fragments(S, rx, x, 0, 0, fx.hi.p, fx.lo.p, three ? fx.mid.p : nullptr);
  to_fragments(S, rb, b, 1, mult_type == 2 ? 1 : 0, fb.hi.p, fb.lo.p, three ? fb.mid.p : nullptr);
  RangeIndex& O = *S.ranges[MP.out_range];
  if (O.nnz == 0) return;
  TCArgs M;
  M.n_out = O.nnz;
  M.ptr = MP.ptr;
  M.pairs = MP.pairs;
  M.xa_hi = fx.hi.p; M.xa_lo = fx.lo.p; M.xa_mid = fx.mid.p;
  M.bb_hi = fb.hi.p; M.bb_lo = fb.lo.p; M.bb_mid = fb.mid.p;
  M.o_row = O.nb_row.p; M.o_cover = O.nb_cover.p; M.o_elem = O.nb_elem.p;
  M.prim_nsf = S.dg.prim_nsf.p; M.cover_nsf = S.dg.cover_nsf.p;
  M.out = out;
  const int grid = (int)(((int64_t)M.n_out * 32 + 127) / 128);
  if (three) k_mult_split3<<<grid, 128, 0, S.stream>>>(M);
  else k_mult_split2<<<grid, 128, 0, S.stream>>>(M);
  S.launches++;
  CQ_CUDA(cudaGetLastError());
}

// Kernel choice of a two-part split product: the system's setting, or (setting -1) a fixed rule on the product's counts,
// so that a product always runs the same kernel (and gives the same bits) whatever else runs on the device.  Two costs
// are compared:
//  - a block per mma.sync warp: 18 us and a time per pair, which is that of the 2 KB of fragments it fetches: 105 to
//    118 ps with B's fragments (1 KB per block) well inside the L2, 125 to 151 ps where they are as large as it, 148 ps at
//    four times its size (112, 143 and 148 below);
//  - tcgen05 tiles: 40 us and the tensor work they issue, at 690 to 890 TFLOP/s once there are a few hundred tiles
//    (820 below).
// The tiles are taken only where at least kTileMinFill of that work is useful: the bound that this choice has always had
// (dense products of 4 x 4 blocks lie under it and would gain: 2288 / 208 us on a 300-atom cluster at 32 bohr).
// Measured in us, blocks / tiles: LS.L -> LSL of DZP cells (26, 16 -> 42 bohr) 216 atoms 1549 / 2162, 512 atoms 4004 /
// 4897, 1000 atoms 9267 / 8615, 1728 atoms 16655 / 14643, 4096 atoms 40,200 / 39,500; 20, 20 -> 40 bohr 512 atoms 5439 / 5040, 1000 atoms 10891 / 8941;
// 300-atom clusters (16, 16) 236 / 270, (20, 20) 594 / 499, (32, 32) 2387 / 1252, and of 4- and 13-orbital atoms
// 2318 / 470; 100 atoms (16, 16) 55 / 66, (20, 20) 91 / 79.
constexpr double kTileMinFill = 0.11;
constexpr int64_t kTileMinPairs = 300000;     // fewer never pay: no estimate of the tiles' work is made

bool split_tiles_pay(int64_t n_pairs, int64_t flops, double issued_flops, int64_t b_blocks) {
  if (n_pairs < kTileMinPairs || issued_flops <= 0.0 || 3.0 * (double)flops < kTileMinFill * issued_flops) return false;
  const double mb = (double)b_blocks * 1024e-6;
  auto part = [&](double from, double to) { return std::min(std::max((mb - from) / (to - from), 0.0), 1.0); };
  const double ps = 112.0 + 31.0 * part(64.0, 127.0) + 5.0 * part(127.0, 500.0);
  return 40e-6 + issued_flops / 820e12 < 18e-6 + (double)n_pairs * ps * 1e-12;
}

void mat_mult_mixed(System& S, int mult_type, int ra, int rb, int rc, double* a, const double* b, double* c,
                    int parts) {
  MixedPlan& MP = get_mixed_plan(S, mult_type, ra, rb, rc);
  int k = S.mixed_kernel;
  if (parts == 3) k = 1;
  if (k == 0 && !umma_usable(S)) k = 1;
  if (k < 0 && MP.kernel < 0 && capturing(S)) k = 1;   // the estimate below waits for the stream: no choice is recorded
  if (k < 0) {
    if (MP.kernel < 0) {
      MP.kernel = 1;
      if (MP.n_pairs >= kTileMinPairs && umma_usable(S) &&
          split_tiles_pay(MP.n_pairs, MP.flops, umma_issued_estimate(S, mult_type, ra, rb, rc), S.ranges[rb]->nnz))
        MP.kernel = 0;
    }
    k = MP.kernel;
  }
  MP.last = k;
  if (k == 0) mat_mult_umma(S, mult_type, ra, rb, rc, a, b, c);
  else mat_mult_mma_sync(S, MP, mult_type, ra, rb, rc, a, b, c, parts);
}

}  // namespace cqb
