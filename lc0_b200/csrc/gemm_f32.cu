// Products and 3x3 convolutions of the fp32 verification mode on tensor cores.
//
// Every fp32 operand is cut into three bf16 pieces, x = x1 + x2 + x3, each the rounding of what the ones before it leave.  bf16 has
// eight significant bits, so x2 is at most 2^-8 and x3 at most 2^-17 of |x|, and from 2^-110 up the three hold all 24 bits; of a
// smaller x what lies below bf16's last subnormal, 2^-133, is lost (outputs of operands of 1e-35 keep 18 bits).  A product of two
// pieces is exact in fp32, and of the nine six are summed:
//   a1 w1                      order 1
//   a1 w2 + a2 w1              order 2^-8
//   a1 w3 + a2 w2 + a3 w1      order 2^-16
// What is left out (a2 w3 + a3 w2 + a3 w3) is below 2^-23.99 of |a||w|, and comes to 2^-24.04.
// The tensor core adds to its accumulator with truncation, which over a long K range would cost more digits than an FMA chain
// has to lose.  So the sums of order 1 stay in tensor memory for 32 k only and are then added, rounded, in registers.  The small
// orders stay there for the whole range: 20 truncations per 64 k, each below 2^-23 of a sum that is below 2^-6.9 of sum |a||w|,
// i.e. at most 2^-25.6 of sum |a||w| per 64 k where all terms have one sign.  A long K over few columns is summed in two to eight
// pieces (f32_pieces), each with its small orders, by a CTA of a cluster each or in turn.  A row's sum is taken in the same order at
// every number of rows and grid.
// Error against sums in 64 bits (relative 2-norm), this kernel / FMA kernel (convolutions: the FMA kernel on the gathered taps), of
// operands as the networks have them (weights of both signs):
//   normal operands    1024x1024x256 0.68e-7 / 1.5e-7   1024x3072x1024 0.95e-7 / 2.9e-7   512x1024x1536 1.1e-7 / 2.5e-7
//                      128x512x4096 1.0e-7 / 3.0e-7   convolutions 112 -> 128 0.82e-7 / 1.5e-7   256 -> 256 0.89e-7 / 2.2e-7
//   non-negative A     the same within 5 %
// Where one sign or one term prevails the FMA kernel can be the better one: both operands non-negative, 1024x3072x1024
// 0.81e-7 / 1.3e-7, 512x1024x1536 0.80e-7 / 0.77e-7, 128x512x4096 0.63e-7 / 0.79e-7, convolution 256 -> 256 0.61e-7 / 0.68e-7;
// operands over eight decades 0.1e-7 .. 1.3e-7 / 0.1e-7 .. 1.2e-7; every operand 1 + 2^-8 - 2^-17 + 2^-23 (the most that can be
// left out), 1536 k in one piece 1.4e-7 / 1.0e-7.
// With 64 k per rounded sum 1024x3072x1024 had 1.04e-7.
//
// The FMA pipe has 74 TFLOP/s and gave half of them; six MMAs for one leave 277 at the measured bf16 rate.  What paces a
// k-block of 64 columns (0.67 us alone on an SM, its MMAs 0.40, its shared-memory traffic 0.55): waits of the issuing thread,
// some 150 cycles each, which the queue of MMAs hides only in part; and what a tile has beside its k-blocks, about 7 us of
// prologue, first loads and epilogue (4.8 at 32 columns), which nothing covers, since a CTA has one tile: 38 % of it at K =
// 1024.  Hence one wait for A and one for the accumulators per k-block and nothing else.  A's pieces live in tensor memory,
// where an MMA reads them beside shared memory; in shared memory (48 KB written and 64 KB read more per k-block) it took 0.79
// us at 64 columns and 1.25 at 128.  Twice as many converter warps were slower (0.80), waits between the MMAs too. us per
// launch, FMA kernel / this: 1024x3072x1024 175 / 56, 1024x1024x1024 70 / 19, 64x1024x1024 13 / 13, 4096x3072x1024 678 / 198;
// 3x3 convolution 128 -> 128 of 64 boards 53 / 16.3.
//   warp 8       TMA: fp32 tile of A, pieces of W (made once at load); the weights' first stages ahead of the grid dependency
//   warps 0-7    fp32 rows (a thread has one row, half of 64 k) -> three bf16 pieces -> tensor memory
//   warp 9       tcgen05.mma (cta_group::1, A from tensor memory)
//   warps 10-17  after every k-block: order-1 sums of its halves -> added in registers; at the end the small orders, then through
//                shared memory to whole rows: scale, bias, activation, skip
// Infinities: inf times a piece that is zero would be NaN, and a value may round to an infinite piece; an output that comes
// out non-finite is therefore computed again from the fp32 operands, by FMAs.
// Every wait is bounded like those of gemm_tc.cu.
#include <atomic>

#include "kernels.cuh"
#include "tcgen05.cuh"

namespace b200 {
namespace {

constexpr int kF32Threads = 18 * 32;
constexpr int kAStages = 2;

struct F32Params {
  const float* A; long long lda;
  const float* W; long long ldw;
  const float* bias;
  float* C; long long ldc;
  const float* skip; long long ldskip;
  int M, N, K, act;
  float scale, alpha;
  int conv_cin;   // convolution: A is [M][cin] on 8x8 boards, W [9][N][cin]
  int cblocks;    // ... k-blocks per tap
  int k_blocks;
  int pieces;     // of K, each summed by itself; see f32_pieces
  int vec_c;      // C may be written, skip and bias read in 16-byte pieces
  int* status;
};

// What a CTA does with the pieces of K: there is one; it takes them in turn; a CTA of a cluster takes each.
enum F32Pieces { kOnePiece, kInTurn, kCluster };

template <int BN> struct F32Tile {
  static constexpr int kRaw = 128 * 64 * 4, kW = 3 * BN * 128;  // bytes of a k-block: two boxes of 32 fp32 columns, pieces of W
  static constexpr int kStage = kRaw + kW;
  static constexpr int kStages = BN == 64 ? 3 : 4;
  static constexpr int kOut = 128 * (BN + 4) * 4;  // the tile's sums, in place of the ring
  // sums of the pieces so far: of 32 columns in registers; 64 would not leave enough of those and have room behind the ring
  static constexpr bool kOutBehind = BN > 32;
  static constexpr int kBytes = kStages * kStage + 1024 /*alignment*/ + 256 /*barriers*/;
  static constexpr int bytes(F32Pieces mode) { return kBytes + (mode == kInTurn && kOutBehind ? kOut : 0); }
  static_assert(kStages * kStage >= kOut, "the sums take the place of the ring");
  // tensor memory: two buffers for the order-1 sums of either half of a k-block, one or two for the small orders (BN columns each),
  // stages of A's pieces (for either half of the k-block 3 x 16 columns)
  static constexpr int kXBufs = BN == 32 ? 2 : 1;
  static constexpr int kXCol = 4 * BN, kACol = (4 + kXBufs) * BN, kCols = 512;
  static_assert(kACol + kAStages * 96 <= kCols, "tensor memory");
};

// D += A W^T with A in tensor memory (one row per lane, two values of k per column).
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t wdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(wdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The three bf16 pieces of two values (the first in the lower half).
__device__ __forceinline__ void split3(float x, float y, uint32_t& u1, uint32_t& u2, uint32_t& u3) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u1) : "f"(y), "f"(x));
  x = __fsub_rn(x, __uint_as_float(u1 << 16));
  y = __fsub_rn(y, __uint_as_float(u1 & 0xffff0000u));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u2) : "f"(y), "f"(x));
  x = __fsub_rn(x, __uint_as_float(u2 << 16));
  y = __fsub_rn(y, __uint_as_float(u2 & 0xffff0000u));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u3) : "f"(y), "f"(x));
}

// W [count] -> planes [3][count]
__global__ void __launch_bounds__(256) split_weights_kernel(const float* __restrict__ w, long long count, __nv_bfloat16* __restrict__ out) {
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i >= count) return;
  uint32_t u1, u2, u3;
  split3(w[i], 0.f, u1, u2, u3);
  out[i] = __ushort_as_bfloat16((unsigned short)u1);
  out[count + i] = __ushort_as_bfloat16((unsigned short)u2);
  out[2 * count + i] = __ushort_as_bfloat16((unsigned short)u3);
}

__device__ __forceinline__ float4 add_rn(const float4 a, const float4 b) {
  return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}
// The four numbers at `q`'s place in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ float4 load_peer(const float* q, int rank) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(mapa(smem_u32(q), (uint32_t)rank)) : "memory");
  return v;
}

// Row m, column n of the product from the fp32 operands, by a whole warp.
template <bool kConv>
__device__ __forceinline__ float warp_dot(const F32Params& p, int m, int n) {
  const int lane = threadIdx.x & 31;
  float v = 0.f;
  if constexpr (kConv) {
    for (int t = 0; t < 9; ++t) {
      const int y = ((m >> 3) & 7) + t / 3 - 1, x = (m & 7) + t % 3 - 1;
      if ((unsigned)y >= 8u || (unsigned)x >= 8u) continue;
      const float* a = p.A + (long long)(m + (t / 3 - 1) * 8 + t % 3 - 1) * p.conv_cin;
      const float* w = p.W + ((long long)t * p.N + n) * p.conv_cin;
      for (int k = lane; k < p.conv_cin; k += 32) v = fmaf(a[k], w[k], v);
    }
  } else {
    for (int k = lane; k < p.K; k += 32) v = fmaf(p.A[m * p.lda + k], p.W[n * p.ldw + k], v);
  }
  return warp_sum(v);
}

template <int BN, bool kConv, F32Pieces kMode>
__global__ void __launch_bounds__(kF32Threads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const F32Params p) {
  using L = F32Tile<BN>;
  constexpr int S = L::kStages, AS = kAStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S * L::kStage);  // [S] A and W have landed
  uint64_t* empty_bar = full_bar + S;                                      // [S] read by eight converter warps and the MMAs
  uint64_t* afull_bar = empty_bar + S;                                     // [AS] pieces of A in place (eight warps)
  uint64_t* aempty_bar = afull_bar + AS;                                   // [AS] ... and read by the MMAs
  uint64_t* hfull_bar = aempty_bar + AS;                                   // [2] order-1 sums complete
  uint64_t* hempty_bar = hfull_bar + 2;                                    // [2] ... and read by eight warps
  uint64_t* xfull_bar = hempty_bar + 2;                                    // [kXBufs] every MMA of a piece of K done
  uint64_t* xempty_bar = xfull_bar + L::kXBufs;                            // [kXBufs] its small orders read by eight warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xempty_bar + L::kXBufs);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int ks = kMode == kCluster ? p.pieces : 1, rank = kMode == kCluster ? (int)blockIdx.x % ks : 0;
  const int n0 = (int)blockIdx.x / ks * BN, m0 = (int)blockIdx.y * 128;
  // this CTA's k-blocks [kb0, kb0 + kbn) and where its q-th piece of them ends
  const int kb0 = kMode == kCluster ? rank * p.k_blocks / ks : 0;
  const int kbn = kMode == kCluster ? (rank + 1) * p.k_blocks / ks - kb0 : p.k_blocks;
  const int nq = kMode == kInTurn ? p.pieces : 1;
  auto piece_end = [&](int q) { return kMode == kInTurn ? (q + 1) * kbn / nq : kbn; };

  if (tid == 256) {
    tma_prefetch_map(&tmap_w);
    tma_prefetch_map(&tmap_a);
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 1);
      mbar_init(smem_u32(&empty_bar[i]), 9);
    }
    for (int i = 0; i < AS; ++i) {
      mbar_init(smem_u32(&afull_bar[i]), 8);
      mbar_init(smem_u32(&aempty_bar[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&hfull_bar[i]), 1);
      mbar_init(smem_u32(&hempty_bar[i]), 8);
    }
    for (int i = 0; i < L::kXBufs; ++i) {
      mbar_init(smem_u32(&xfull_bar[i]), 1);
      mbar_init(smem_u32(&xempty_bar[i]), 8);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)L::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  // after the allocation: the next kernel's CTAs must not take the tensor memory that this one still waits for
  grid_launch_dependents();
  const uint32_t tmem = *tmem_slot;
  float* out = reinterpret_cast<float*>(kMode == kInTurn && L::kOutBehind ? smem + S * L::kStage + 256 : smem);

  if (warp < 8) {
    // ---------------- A: fp32 rows -> pieces ----------------
    const int quarter = warp & 3, half = warp >> 2, row = quarter * 32 + lane;
    const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + L::kACol + half * 48;
    int s = 0, a = 0;
    uint32_t ph = 0, aph = 0;
    for (int i = 0; i < kbn; ++i) {
      if (!mbar_wait(smem_u32(&full_bar[s]), ph, abort_flag, 1)) break;
      const uint8_t* src = smem + s * L::kStage + half * 16384 + row * 128;
      float v[32];
#pragma unroll
      for (int c = 0; c < 8; ++c) *reinterpret_cast<float4*>(v + 4 * c) = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&empty_bar[s]));
      if (++s == S) { s = 0; ph ^= 1; }
      if (i >= AS && !mbar_wait(smem_u32(&aempty_bar[a]), aph ^ 1, abort_flag, 2)) break;
      tcgen05_fence_after();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t u[3][8];
#pragma unroll
        for (int c = 0; c < 8; ++c) split3(v[16 * h + 2 * c], v[16 * h + 2 * c + 1], u[0][c], u[1][c], u[2][c]);
#pragma unroll
        for (int c = 0; c < 3; ++c) tmem_st8(ta + a * 96 + c * 16 + h * 8, u[c]);
      }
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&afull_bar[a]));
      if (++a == AS) { a = 0; aph ^= 1; }
    }
  } else if (warp == 8) {
    // ---------------- TMA ----------------
    if (elect_one()) {
      auto load_w = [&](int i, int s) {
        const uint32_t fb = smem_u32(&full_bar[s]), dst = smem_u32(smem + s * L::kStage) + L::kRaw;
        mbar_expect_tx(fb, L::kStage);
        int row = n0, x = (kb0 + i) * 64, plane = p.N;
        if constexpr (kConv) {
          const int tap = (kb0 + i) / p.cblocks;
          x = (kb0 + i - tap * p.cblocks) * 64;
          row += tap * p.N;
          plane = 9 * p.N;
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) tma_load_2d(dst + j * BN * 128, &tmap_w, x, row + j * plane, fb);
      };
      // loaded weights: requested while the kernel before this one is still running
      const int early = kbn < S ? kbn : S;
      for (int i = 0; i < early; ++i) load_w(i, i);
      grid_dependency_wait();
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < kbn; ++i) {
        if (i >= early) {
          if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag, 3)) break;
          load_w(i, s);
        }
        const uint32_t fb = smem_u32(&full_bar[s]), dst = smem_u32(smem + s * L::kStage);
        if constexpr (kConv) {
          const int tap = (kb0 + i) / p.cblocks, x = (kb0 + i - tap * p.cblocks) * 64;
#pragma unroll
          for (int h = 0; h < 2; ++h) tma_load_4d(dst + h * 16384, &tmap_a, x + 32 * h, tap % 3 - 1, tap / 3 - 1, m0 >> 6, fb);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) tma_load_2d(dst + h * 16384, &tmap_a, (kb0 + i) * 64 + 32 * h, m0, fb);
        }
        if (++s == S) { s = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t one = make_idesc<__nv_bfloat16, BN>();
      bool good = true;
      int s = 0, i = 0;
      for (int q = 0; q < nq && good; ++q) {
        const int first = i, end = piece_end(q), xb = q % L::kXBufs;
        // the small orders of the piece that had this buffer have been read
        if (q >= L::kXBufs && !mbar_wait(smem_u32(&xempty_bar[xb]), (q / L::kXBufs - 1) & 1, abort_flag, 9)) { good = false; break; }
        for (; i < end; ++i) {
          // A's pieces are in place; the warps that wrote them have seen the weights land too
          if (!mbar_wait(smem_u32(&afull_bar[i & 1]), (i >> 1) & 1, abort_flag, 5)) { good = false; break; }
          if (i > 1 && !mbar_wait(smem_u32(&hempty_bar[i & 1]), ((i >> 1) & 1) ^ 1, abort_flag, 6)) { good = false; break; }
          tcgen05_fence_after();
          const int a = i & 1;
          const uint32_t sw = smem_u32(smem + s * L::kStage) + L::kRaw, a1 = tmem + L::kACol + a * 96;
          const uint32_t h = tmem + a * 2 * BN, x = tmem + L::kXCol + xb * BN;
          const uint64_t w1 = make_smem_desc(sw), w2 = make_smem_desc(sw + BN * 128), w3 = make_smem_desc(sw + 2 * BN * 128);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_ts(h + (k >> 1) * BN, a1 + (k >> 1) * 48 + 8 * (k & 1), w1 + 2 * k, one, (k & 1) ? 1u : 0u);
          tcgen05_commit(smem_u32(&hfull_bar[a]));
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t ak = a1 + (k >> 1) * 48 + 8 * (k & 1);
            mma_ts(x, ak, w3 + 2 * k, one, (i > first || k > 0) ? 1u : 0u);
            mma_ts(x, ak + 16, w2 + 2 * k, one, 1u);
            mma_ts(x, ak + 32, w1 + 2 * k, one, 1u);
            mma_ts(x, ak, w2 + 2 * k, one, 1u);
            mma_ts(x, ak + 16, w1 + 2 * k, one, 1u);
          }
          tcgen05_commit(smem_u32(&aempty_bar[a]));
          tcgen05_commit(smem_u32(&empty_bar[s]));
          if (++s == S) s = 0;
        }
        if (good) tcgen05_commit(smem_u32(&xfull_bar[xb]));
      }
    }
    __syncwarp();
  } else {
    // ---------------- sums ----------------
    // a thread has one row, half of the columns
    constexpr int kCols = BN / 2;
    const int quarter = warp & 3, half = (warp - 10) >> 2;
    const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + half * kCols;
    constexpr bool kKeep = kMode == kInTurn && !L::kOutBehind;
    float acc[kCols], tot[kKeep ? kCols : 1];
    float* row = out + (quarter * 32 + lane) * (BN + 4) + half * kCols;
    bool good = true;
    for (int q = 0, i = 0; q < nq && good; ++q) {
      const int end = piece_end(q), xb = q % L::kXBufs;
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
      for (; i < end; ++i) {
        const int b = i & 1;
        if (!mbar_wait(smem_u32(&hfull_bar[b]), (i >> 1) & 1, abort_flag, 7)) { good = false; break; }
        tcgen05_fence_after();
#pragma unroll
        for (int c = 0; c < kCols; c += 16) {
          uint32_t r0[16], r1[16];
          tmem_ld16(ta + 2 * b * BN + c, r0);
          tmem_ld16(ta + (2 * b + 1) * BN + c, r1);
          tmem_ld_wait();
          if (c + 16 >= kCols) {  // the last columns are in registers: the k-block after the next may overwrite them
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&hempty_bar[b]));
          }
#pragma unroll
          for (int k = 0; k < 16; ++k)
            acc[c + k] = __fadd_rn(acc[c + k], __fadd_rn(__uint_as_float(r0[k]), __uint_as_float(r1[k])));
        }
      }
      if (good) good = mbar_wait(smem_u32(&xfull_bar[xb]), (q / L::kXBufs) & 1, abort_flag, 8);
      tcgen05_fence_after();
      // the piece's sums, the small orders last
#pragma unroll
      for (int c = 0; c < kCols; c += 16) {
        uint32_t x[16];
        tmem_ld16(ta + L::kXCol + xb * BN + c, x);
        tmem_ld_wait();
        if (kMode == kInTurn && c + 16 >= kCols) {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&xempty_bar[xb]));
        }
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          float4 v = make_float4(__fadd_rn(acc[c + j], __uint_as_float(x[j])), __fadd_rn(acc[c + j + 1], __uint_as_float(x[j + 1])),
                                 __fadd_rn(acc[c + j + 2], __uint_as_float(x[j + 2])), __fadd_rn(acc[c + j + 3], __uint_as_float(x[j + 3])));
          if constexpr (kKeep) {
            if (q > 0) v = add_rn(make_float4(tot[c + j], tot[c + j + 1], tot[c + j + 2], tot[c + j + 3]), v);
            tot[c + j] = v.x; tot[c + j + 1] = v.y; tot[c + j + 2] = v.z; tot[c + j + 3] = v.w;
          } else {
            if (kMode == kInTurn && q > 0) v = add_rn(*reinterpret_cast<const float4*>(row + c + j), v);
            *reinterpret_cast<float4*>(row + c + j) = v;  // where the ring was, which is free after the only piece, or behind it
          }
        }
      }
    }
    if constexpr (kKeep) {
#pragma unroll
      for (int c = 0; c < kCols; c += 4) *reinterpret_cast<float4*>(row + c) = make_float4(tot[c], tot[c + 1], tot[c + 2], tot[c + 3]);
    }
    tcgen05_fence_before();
    if constexpr (kMode != kCluster) asm volatile("bar.sync 1, 256;" ::: "memory");
  }
  auto free_tmem = [&] {
    if (warp == 9) {
      tcgen05_fence_after();
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)L::kCols) : "memory");
    }
    __syncwarp();
  };
  if constexpr (kMode == kCluster) {
    // The sums of the others' pieces.  Tensor memory is given back ahead of the wait for them: an SM of theirs may be held by a
    // cluster of another network's kernel that waits for this one's.
    __syncwarp();
    tcgen05_fence_before();
    __syncthreads();
    free_tmem();
    cluster_sync_all();
  }

  if (warp >= 10) {
    grid_dependency_wait();  // the residual input
    const int t = tid - 320;
#pragma unroll 1
    for (int e = t * 4 + rank * 1024; e < 128 * BN; e += 1024 * ks) {  // the CTAs of a cluster take turns
      const int r = e / BN, c = e % BN, m = m0 + r, n = n0 + c;
      const bool in = m < p.M && n < p.N;
      const float* mine = out + r * (BN + 4) + c;
      float4 q = *reinterpret_cast<const float4*>(mine);
      if (kMode == kCluster && in) {
        q = load_peer(mine, 0);
        for (int j = 1; j < ks; ++j) q = add_rn(q, load_peer(mine, j));
      }
      float v[4] = {q.x, q.y, q.z, q.w};
      bool again = false;
#pragma unroll
      for (int j = 0; j < 4; ++j) again |= in && n + j < p.N && !(fabsf(v[j]) <= 3.402823466e38f);
      for (uint32_t todo = __ballot_sync(0xffffffffu, again); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const int mm = __shfl_sync(0xffffffffu, m, src), nn = __shfl_sync(0xffffffffu, n, src);
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          const float d = nn + j < p.N ? warp_dot<kConv>(p, mm, nn + j) : 0.f;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (lane == src && k == j) v[k] = d;
        }
      }
      if (!in) continue;
      const bool whole = p.vec_c && n + 4 <= p.N;
      float b4[4] = {0.f, 0.f, 0.f, 0.f}, s4[4] = {0.f, 0.f, 0.f, 0.f};
      const float* skip = p.skip ? p.skip + (long long)m * p.ldskip + n : nullptr;
      if (whole) {
        if (p.bias) *reinterpret_cast<float4*>(b4) = __ldg(reinterpret_cast<const float4*>(p.bias + n));
        if (skip) *reinterpret_cast<float4*>(s4) = *reinterpret_cast<const float4*>(skip);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (p.bias && n + j < p.N) b4[j] = __ldg(p.bias + n + j);
          if (skip && n + j < p.N) s4[j] = skip[j];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] *= p.scale;
        if (p.bias) v[j] += b4[j];
        v[j] = activate<false>(v[j], p.act);
        if (skip) v[j] = p.alpha * v[j] + s4[j];
      }
      float* o = p.C + (long long)m * p.ldc + n;
      if (whole) {
        *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < p.N) o[j] = v[j];
      }
    }
  }
  __syncwarp();
  if constexpr (kMode == kCluster) {
    cluster_sync_all();  // the others have read this CTA's sums
  } else {
    tcgen05_fence_before();
    __syncthreads();
    free_tmem();
  }
  if (*abort_flag) {
    // Give copies that may still be in flight time to land before the CTA's shared memory is released.
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    if (tid == 0 && p.status) atomicCAS(p.status, 0, 600 + *abort_flag);
  }
}

template <int BN, bool kConv, F32Pieces kMode>
cudaError_t launch_f32_bn(const F32Params& p, const void* planes, cudaStream_t s) {
  using L = F32Tile<BN>;
  cudaError_t e = raise_smem_limit<&gemm_f32_kernel<BN, kConv, kMode>>(L::bytes(kMode));
  if (e != cudaSuccess) return e;
  CUtensorMap ma, mw;
  if ((e = gemm_f32_map(p.A, p.lda, p.M, kConv ? p.conv_cin : p.K, kConv, &ma)) != cudaSuccess) return e;
  const int rows = 3 * (kConv ? 9 : 1) * p.N, cols = kConv ? p.conv_cin : p.K;
  if ((e = gemm_tensor_map(planes, cols, rows, cols, BN, TypeTag<__nv_bfloat16>::prec, &mw)) != cudaSuccess) return e;
  const int ks = kMode == kCluster ? p.pieces : 1;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(ceil_div(p.N, BN) * ks, ceil_div(p.M, 128));
  lc.blockDim = dim3(kF32Threads);
  lc.dynamicSmemBytes = L::bytes(kMode);
  lc.stream = s;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (kMode == kCluster) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = ks;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (t_dependent_launch) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  lc.attrs = attr;
  lc.numAttrs = na;
  return cudaLaunchKernelEx(&lc, gemm_f32_kernel<BN, kConv, kMode>, ma, mw, p);
}

// Pieces that K is summed in, from N and K alone, so that a row's sum is the same in every batch: one to about nine k-blocks where the
// columns are so few that the tiles of a small batch leave most SMs idle.  fp32 networks, us, FMA kernel / one piece / pieces: 20 x 256
// residual 1 board 1131 / 1282 / 616, 3 1156 / 1332 / 631, 8 1674 / 1340 / 664; 10 x 128 4 boards 405 / 418 / 308; three blocks of
// 512 filters 1 board 467 / 664 / 370.  Taken in turn they cost a few per cent where the tiles fill the GPU (20 x 256, 64
// boards 7485 / 1724 / 1774; 10 x 128 1315 / 458 / 468).
int f32_pieces(int N, int k_blocks) {
  return N > 512 || k_blocks < 18 ? 1 : k_blocks < 36 ? 2 : k_blocks < 72 ? 4 : 8;
}


// Tile width: rounds of tiles (one per SM) times a tile's time, its k-blocks and its ends in ns.  Measured at 32 / 64 columns, us:
// 64x1024x1024 13.0 / 16.3, 1024x1024x1024 28.0 / 19.6, 1024x1024x1536 37.1 / 25.4, 1024x3072x1024 82 / 56, 512x4096x256 27.8 / 19.8,
// convolution of 64 boards 16.3 / 20.7, of 512 111 / 82.
template <bool kConv>
cudaError_t launch_f32(F32Params& p, const void* planes, int sm_count, cudaStream_t s) {
  const long long m_tiles = ceil_div(p.M, 128);
  auto cost = [&](int bn, int block, int ends) {
    return ceil_div(m_tiles * ceil_div(p.N, bn), sm_count) * ((long long)p.k_blocks * block + ends);
  };
  p.pieces = f32_pieces(p.N, p.k_blocks);
  const bool narrow = cost(32, 525, 4800) < cost(64, 700, 7000);
  if (p.pieces == 1)
    return narrow ? launch_f32_bn<32, kConv, kOnePiece>(p, planes, s) : launch_f32_bn<64, kConv, kOnePiece>(p, planes, s);
  // clusters while the tiles of 32 columns times the pieces are one round (an eighth of the SMs may not form whole clusters)
  if (m_tiles * ceil_div(p.N, 32) * p.pieces <= sm_count - sm_count / 8) return launch_f32_bn<32, kConv, kCluster>(p, planes, s);
  return narrow ? launch_f32_bn<32, kConv, kInTurn>(p, planes, s) : launch_f32_bn<64, kConv, kInTurn>(p, planes, s);
}

bool al16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

}  // namespace

cudaError_t launch_split_weights(const float* w, long long count, void* planes, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  split_weights_kernel<<<ceil_div(count, 256), 256, 0, s>>>(w, count, static_cast<__nv_bfloat16*>(planes));
  return cudaGetLastError();
}

bool gemm_f32_supported(const GemmParams& g) {
  const int k = g.conv_cin > 0 ? g.conv_cin : g.K;
  return g.W3 && g.batch == 1 && g.batch_rows == 0 && k >= 8 && (k % 8) == 0 && (g.lda % 4) == 0 && (g.conv_cin > 0 || g.ldw == g.K) &&
         al16(g.A) && al16(g.W3) && !g.a_stats && !g.res && !g.out_stats && g.n_split == 0 && g.se_k == 0 && !g.ln_gamma;
}

cudaError_t launch_gemm_f32(const GemmParams& g, int* status, int sm_count, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0) return cudaSuccess;
  if (!gemm_f32_supported(g)) return cudaErrorInvalidValue;
  F32Params p = {};
  p.A = static_cast<const float*>(g.A); p.lda = g.conv_cin > 0 ? g.conv_cin : g.lda;
  p.W = static_cast<const float*>(g.W); p.ldw = g.ldw;
  p.bias = g.bias;
  p.C = static_cast<float*>(g.C); p.ldc = g.ldc;
  p.skip = static_cast<const float*>(g.skip); p.ldskip = g.ldskip;
  p.M = g.M; p.N = g.N; p.K = g.K; p.act = g.act; p.scale = g.scale; p.alpha = g.alpha;
  p.conv_cin = g.conv_cin;
  p.cblocks = ceil_div(g.conv_cin, 64);
  p.k_blocks = g.conv_cin > 0 ? 9 * p.cblocks : ceil_div(g.K, 64);
  p.vec_c = al16(g.C) && g.ldc % 4 == 0 && (!g.skip || (al16(g.skip) && g.ldskip % 4 == 0)) && (!g.bias || al16(g.bias));
  p.status = status;
  return g.conv_cin > 0 ? launch_f32<true>(p, g.W3, sm_count, s) : launch_f32<false>(p, g.W3, sm_count, s);
}

}  // namespace b200
