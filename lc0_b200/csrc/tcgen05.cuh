// Building blocks shared by the tcgen05 kernels (gemm_tc.cu, gemm_split.cu): PTX wrappers of mbarriers, TMA, tensor
// memory and tcgen05.mma, operand and instruction descriptors, and the parameter block of their epilogues.
#pragma once
#include <cuda.h>

#include "kernels.cuh"

namespace b200 {
namespace {

constexpr int BM = 128;
constexpr int BK = 64;  // 64 16-bit elements = one 128-byte swizzle row
constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // 2 s

// ---- PTX wrappers ------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// One lane of a converged warp.  The warp that issues TMA or tcgen05 instructions picks its lane with this and not with a lane
// index: the compiler then knows that a single thread runs the block and keeps the instructions' operands in uniform
// registers.  With `lane == 0` a k-block of four MMAs took 731 cycles to issue, with the election 495.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok));
  return ok != 0;
}
// Index of this thread's warp, known to the compiler to be the same in the whole warp.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
// Same with a suspend-time hint: the thread may sleep in hardware for up to `ns` nanoseconds (it is woken when the
// phase completes), so a long wait costs few issue slots of the warps that share its scheduler.
__device__ __forceinline__ uint32_t mbar_try_wait_hint(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(ns)
      : "memory");
  return ok;
}
// Bounded wait.  Returns false when the CTA is aborting (this or another role timed out).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0 = 0;  // the clock is first read after 64 tries: reading it is slow
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait_hint(bar, parity, 20000u)) return true;
    if ((it & 63) == 0) {
      if (*abort_flag) return false;
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > kWaitLimitNs) {
        *abort_flag = code;
        return false;
      }
    }
  }
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// 4D tile load (channels, file, rank, position); coordinates may lie outside the tensor, those elements are
// zero-filled, which is exactly the zero padding of a same-padded convolution on the 8x8 board.
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
// Brings a tensor map into the descriptor cache ahead of its first use (the first TMA store of a launch otherwise
// waited about three microseconds for it).
__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Waits until at most one of this thread's bulk groups still reads its shared-memory source.
__device__ __forceinline__ void tma_store_wait_read1() {
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_read0() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_all0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void tcgen05_mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }


// ---- CTA-pair (cta_group::2) helpers -------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on a barrier of a CTA of the cluster.  Relaxed: the arrivals of this kernel only hand tensor memory back
// to the MMA issuer (ordered by tcgen05.fence), no generic-proxy data is published through them; a release at
// cluster scope here stalled the arriving thread for 2-3 thousand cycles per tile.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load whose completion is signalled on a barrier that may live in the peer CTA of the pair (no multicast:
// each CTA of the pair fetches its own half of the operands).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                                 uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tcgen05_commit_pair(uint32_t cluster_bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_bar)
               : "memory");
}
// Arrival on the barrier at offset `bar` of both CTAs of the pair once the MMAs issued so far are done.
__device__ __forceinline__ void tcgen05_commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void tcgen05_mma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                     uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile stored as rows of 128 bytes with the 128-byte
// swizzle (what a TMA box of 64 16-bit elements x R rows with CU_TENSOR_MAP_SWIZZLE_128B produces):
// start address >> 4 in bits [0,14), stride between 8-row groups (1024 B) >> 4 in bits [32,46),
// descriptor version 1 in bits [46,48), layout type 2 (SWIZZLE_128B) in bits [61,64).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Activation of a register array with the selection hoisted out of the element loop.
template <int N>
__device__ __forceinline__ void apply_activation(float (&v)[N], int act) {
  switch (act) {
    case ACT_RELU:
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = fmaxf(v[j], 0.f);
      break;
    case ACT_RELU_2:
#pragma unroll
      for (int j = 0; j < N; ++j) { const float t = fmaxf(v[j], 0.f); v[j] = t * t; }
      break;
    case ACT_MISH:
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = mish_f(v[j]);
      break;
    case ACT_SWISH:
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = swish_f(v[j]);
      break;
    case ACT_NONE:
      break;
    default:
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] = activate<true>(v[j], act);
      break;
  }
}

template <typename T> struct FmtCode;
template <> struct FmtCode<__half> { static constexpr uint32_t v = 0; };
template <> struct FmtCode<__nv_bfloat16> { static constexpr uint32_t v = 1; };

// Instruction descriptor of tcgen05.mma.kind::f16: D format fp32 (bits 4-5 = 1), A/B format (bits 7-9,
// 10-12: 0 = f16, 1 = bf16), both operands K-major (bits 15, 16 = 0), N >> 3 in bits 17-22, M >> 4 in bits 24-28.
template <typename T, int BN>
__device__ __forceinline__ constexpr uint32_t make_idesc() {
  return (1u << 4) | (FmtCode<T>::v << 7) | (FmtCode<T>::v << 10) | ((uint32_t)(BN >> 3) << 17) |
         ((uint32_t)(BM >> 4) << 24);
}

struct TcParams {
  const float* bias;
  void* C;
  long long ldc;
  int M, N, K;
  int act;
  float scale, alpha;
  int out_f32;
  int* status;
  int tma_store;  // 1: 16-bit output staged in shared memory and written with TMA stores
  // CTA-pair kernel: the tiles from split_from on are computed as two half-width tiles each (tiles_v virtual tiles in
  // all), so that a last, less than half filled wave spreads over all pairs; split_from >= tiles_v means no split
  int split_from, tiles_v;
  int conv_cblocks;  // > 0: 3x3 convolution, number of 64-channel blocks of the input (k_blocks = 9 * conv_cblocks)
  // folded LayerNorm (see GemmParams)
  const double* a_stats; const float* colsum; float a_inv_c, a_eps;
  const void* res; long long ldres;  // residual input (gemm_split.cu; the kernels of gemm_tc.cu have a tensor map for it)
  int res_mode;  // 0 none, 1 add the residual tile, 2 add the normalised residual tile
  const double* res_stats; const float* res_gamma; const float* res_beta; float res_inv_c, res_eps;
  double* out_stats;
  int n_split;  // > 0: columns from here on are stored through the second output map
  // Squeeze-excitation unit fused into the epilogue of a convolution whose tile holds two whole boards and every
  // output channel (se_k > 0; see GemmParams).
  const float* se_w1; const float* se_b1; const float* se_w2; const float* se_b2; const float* se_bias; int se_k;
  void* C2; long long ldc2;  // second output of gemm_split.cu (the pair kernel has a tensor map for it)
  int vec_c;                 // gemm_split.cu: C (and C2) may be written in 16-byte pieces
  int w_const;               // gemm_split.cu: W may be requested ahead of the grid dependency
  int batch_rows;  // > 0: stacked products, rows [b * batch_rows, (b + 1) * batch_rows) use W rows [b * N, (b + 1) * N)
};

__device__ __forceinline__ void mean_rstd(const double2 st, float inv_c, float eps, float& mean, float& rstd) {
  const double mu = st.x * (double)inv_c;
  const double var = fmax(st.y * (double)inv_c - mu * mu, 0.0);
  mean = (float)mu;
  rstd = rsqrtf((float)var + eps);
}
__device__ __forceinline__ void mean_rstd(const double* stats, long long m, float inv_c, float eps, float& mean, float& rstd) {
  mean_rstd(*reinterpret_cast<const double2*>(stats + 2 * m), inv_c, eps, mean, rstd);
}
// Packs two floats into one 32-bit pair of T; fp16 saturates to the largest finite value.
template <typename T> __device__ __forceinline__ uint32_t pack_pair(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack_pair<__half>(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));  // first source -> upper half
  return r;
}
template <> __device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Epilogue parameters of a product that are the same for every kernel.
inline void fill_tc_params(TcParams& p, const GemmParams& g, int* status) {
  p.bias = g.bias; p.C = g.C; p.ldc = g.ldc;
  p.M = g.M; p.N = g.N; p.K = g.K; p.act = g.act; p.scale = g.scale; p.alpha = g.alpha;
  p.out_f32 = g.out_f32 ? 1 : 0; p.status = status;
  p.tma_store = 0; p.split_from = 0x7fffffff; p.tiles_v = 0;
  p.conv_cblocks = g.conv_cin > 0 ? ceil_div(g.conv_cin, BK) : 0;
  p.a_stats = g.a_stats; p.colsum = g.colsum; p.a_inv_c = g.a_inv_c; p.a_eps = g.a_eps;
  p.res_mode = g.res ? (g.res_stats ? 2 : 1) : 0;
  p.res = g.res; p.ldres = g.ldres;
  p.res_stats = g.res_stats; p.res_gamma = g.res_gamma; p.res_beta = g.res_beta;
  p.res_inv_c = g.res_inv_c; p.res_eps = g.res_eps;
  p.out_stats = g.out_stats;
  p.n_split = g.n_split; p.C2 = g.C2; p.ldc2 = g.ldc2;
  p.se_w1 = g.se_w1; p.se_b1 = g.se_b1; p.se_w2 = g.se_w2; p.se_b2 = g.se_b2; p.se_bias = g.se_bias;
  p.se_k = g.se_k;
  p.batch_rows = g.batch_rows;
  p.w_const = g.w_const ? 1 : 0;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const int per16 = g.out_f32 ? 4 : 8;
  p.vec_c = al16(g.C) && (g.ldc % per16) == 0 && (g.n_split == 0 || (al16(g.C2) && (g.ldc2 % per16) == 0));
}

// Whether the epilogues can take the operands of `g`: statistics, a residual and a second output come with 16-bit rows that TMA
// can write, and the residual with rows that TMA, or a 16-byte load, can read.  The same for every kernel, so that a form is
// taken or refused whatever the number of rows.
inline bool epilogue_supported(const GemmParams& g) {
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const bool folded = g.a_stats || g.res || g.out_stats || g.se_k > 0 || g.n_split > 0;
  if (folded && (g.out_f32 || (g.ldc % 8) != 0 || !al16(g.C))) return false;
  return !g.res || ((g.ldres % 8) == 0 && al16(g.res));
}

}  // namespace

// Tensor map over a row-major 16-bit matrix, box = 64 columns x box_rows, 128-byte swizzle; cached by its arguments.
cudaError_t gemm_tensor_map(const void* ptr, long long ld, int rows, int cols, int box_rows, int prec, CUtensorMap* out);
// Tensor map over fp32 rows, box = 32 columns x 128 rows, 128-byte swizzle; board: over [rows / 64][8][8][cols] (ld ignored), box = 32
// columns x two boards.
cudaError_t gemm_f32_map(const float* ptr, long long ld, int rows, int cols, bool board, CUtensorMap* out);
// Products of few rows (gemm_split.cu).
template <typename T> cudaError_t launch_gemm_split(const GemmParams& g, int* status, int sm_count, cudaStream_t s);

}  // namespace b200
