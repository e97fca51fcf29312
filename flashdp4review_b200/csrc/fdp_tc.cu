// Tensor-core path for bf16 / fp16: one persistent, warp-specialised GEMM kernel template built
// on TMA (cp.async.bulk.tensor, 128-byte swizzle) -> shared-memory ring -> tcgen05.mma with fp32
// accumulators in TMEM -> tcgen05.ld epilogue.  Instances (A major, B major, epilogue, CTAs per tile):
//   wgrad   MN, MN, STORE_SCALED, 2   dW = scale * sum_b c_b G_b^T X_b + noise; every sample's K segment has
//                                     its own TMEM accumulator, added times c_b into registers
//           MN, MN, STORE, 2          same from a pre-scaled copy of G (T < 256, or mostly padded K stages)
//   direct  MN, MN, SUMSQ, 1          per-sample ||G_b^T X_b||_F^2: tile squared in the epilogue, never stored
//   kept    MN, MN, CHAIN_SUMSQ, 2    the same in short chains, the tile kept in the workspace for weighted_sum_kernel; 16-bit
//                                     widths off the multiples of 8 or below 128 have their norms from it in any case
//   gram    K,  K,  GRAM, 1           sum_{t,s} (G_b G_b^T)_{ts} (X_b X_b^T)_{ts}, two accumulators in TMEM
//   dgrad   K,  MN or K, STORE, 2     dX = G W
//   forward K,  K or MN, STORE, 2     Y = X W^T + bias
//           CHAIN_STORE for both       16-bit operands of any width, fp32 output: in short chains
//   fp32    the same products over bf16 parts of the operands: SPLIT_* three products, SPLIT6_* six (SUMSQ, SCALED, STORE)
// Roles in a CTA: warp 0 = TMA producer, warp 1 = MMA issuer and TMEM owner, warps 2-5 (2-9 for the
// store epilogues) = epilogue, each on the TMEM lane quarter warp % 4.  With two CTAs per tile the
// even CTA of a 2-CTA cluster issues tcgen05.mma.cta_group::2 for both.  Every mbarrier wait is
// bounded: when one runs out the CTA records a code in the status word, drains and leaves.
// No TMA load here uses cluster multicast.
#include <cuda.h>
#include <atomic>
#include <cstdlib>
#include <mutex>

#include "fdp_async.cuh"
#include "fdp_gram_units.h"
#include "fdp_kernels.h"

namespace fdp {
namespace {

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4, UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;  // 16 KiB
constexpr int B_STAGE_BYTES = BN * BK * 2;  // 32 KiB
constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
constexpr int BAR_BYTES = 256;
constexpr int BOX_ROWS = 32, BOX_BYTES = BOX_ROWS * 128;   // an epilogue warp's output box: 32 rows of 128 bytes
// EPI_STORE_SCALED keeps the clip factors of up to MAX_SMEM_FACTORS samples in shared memory (what the
// ring and the output boxes leave of the 227 KB); larger batches read them from global memory
constexpr int MAX_SMEM_FACTORS = 384;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + BAR_BYTES;
constexpr int SMEM_BYTES_STORE = SMEM_BYTES + 8 * BOX_BYTES;
constexpr int SMEM_BYTES_SCALED = SMEM_BYTES_STORE + MAX_SMEM_FACTORS * 4;
static_assert(SPLIT_MAXIMA_BYTES % 256 == 0 && SPLIT_MAXIMA_BYTES >= (148 * 16 + 2) * sizeof(unsigned), "a word for every block of tc_split");
static_assert(SMEM_BYTES_SCALED <= 227 * 1024, "shared memory of one CTA");
constexpr int TMEM_COLS = 512;
// Per-sample products kept in a call's workspace.  Beyond that there was nothing to gain: 4 x 2048 rows, 4096 -> 11008 bf16,
// 721 MB of products, a layer's forward and backward 2148 us against 2157 (with the GEMMs before the uniform issue).
constexpr size_t KEEP_LIMIT = static_cast<size_t>(512) << 20;
constexpr int KEEP_SMEM_FACTORS = 128;
constexpr int MAX_SMS = 148;           // workers the split-K parking area is sized for

// EPI_STORE_SCALED: the accumulator of each sample (K segment) is drained on its own and added, times
// that sample's clip factor, to fp32 registers of eight epilogue warps; G needs no scaled copy.
// EPI_SPLIT_*: fp32 inputs as bf16 halves, three products per K stage (see TcArgs::plane_a): the clipped sum,
// a plain product (+ bias), and one sample's product tile squared and summed.
// EPI_SPLIT6_*: the same with bf16 thirds and six products.
// The SUMSQ ones of CTA pairs also keep the tile in HBM for weighted_sum_kernel when TcArgs::keep is set.
// EPI_CHAIN_SUMSQ: one sample's product tile squared and summed for 16-bit operands, in short chains: norms that came from FMA
// kernels before (an accumulator runs for one K stage only; one for all of a sample's stages drifts: 768 rows 6.8e-7, 4000 3.8e-6)
// and products that are kept (kept_chain).
// EPI_CHAIN_STORE: a plain 16-bit product with an fp32 output that FMA kernels computed before, in the same chains.
enum { EPI_STORE = 0, EPI_SUMSQ = 1, EPI_GRAM = 2, EPI_STORE_SCALED = 3, EPI_SPLIT_SCALED = 4, EPI_SPLIT_STORE = 5,
       EPI_SPLIT_SUMSQ = 6, EPI_SPLIT6_SCALED = 7, EPI_SPLIT6_SUMSQ = 8, EPI_SPLIT6_STORE = 9, EPI_CHAIN_SUMSQ = 10, EPI_CHAIN_STORE = 11 };
__host__ __device__ constexpr bool epi_chained(int epi) { return epi >= EPI_STORE_SCALED; }
// bf16 parts of an operand
__host__ __device__ constexpr int epi_planes(int epi) {
  return epi == EPI_SPLIT6_SCALED || epi == EPI_SPLIT6_SUMSQ || epi == EPI_SPLIT6_STORE ? 3 : epi == EPI_SPLIT_SCALED || epi == EPI_SPLIT_STORE || epi == EPI_SPLIT_SUMSQ ? 2 : 1;
}
__host__ __device__ constexpr bool epi_scaled(int epi) { return epi == EPI_STORE_SCALED || epi == EPI_SPLIT_SCALED || epi == EPI_SPLIT6_SCALED; }
__host__ __device__ constexpr bool epi_sumsq(int epi) { return epi == EPI_SPLIT_SUMSQ || epi == EPI_SPLIT6_SUMSQ || epi == EPI_CHAIN_SUMSQ; }
// plain products: bias, tiles cut along N
__host__ __device__ constexpr bool epi_plain(int epi) { return epi == EPI_STORE || epi == EPI_SPLIT_STORE || epi == EPI_SPLIT6_STORE || epi == EPI_CHAIN_STORE; }
__host__ __device__ constexpr bool epi_stores(int epi) { return epi_plain(epi) || epi_scaled(epi); }
// eight epilogue warps (two per TMEM lane quarter, 128 columns each) for the store epilogues, four for the norms
__host__ __device__ constexpr int epi_warps_for(int epi) { return (epi == EPI_STORE || epi_chained(epi)) ? 8 : 4; }
constexpr int threads_for(int epi) { return 64 + 32 * epi_warps_for(epi); }
constexpr int smem_for(int epi) {
  return epi_scaled(epi) ? SMEM_BYTES_SCALED : epi_stores(epi) ? SMEM_BYTES_STORE : SMEM_BYTES;
}

struct TcArgs {
  int M, N;             // extents of the output space of one batch (masks)
  int tiles_m, tiles_n; // tile grid of one batch
  int tiles_per_batch;
  int n_fastest;        // tile order: 1 = consecutive tiles walk along N (keeps the B operand in L2), 0 = along M
  int batch;
  int k_stages, k_stages2;  // K loop of operand pair 1 (and pair 2 for EPI_GRAM)
  int batch_rows;           // rows of one batch along the row coordinate of the tensor maps
  void* out; int out_dt; long long ld_out; float scale; NoiseKey nk;
  float* partials;      // norm passes: one partial per (work unit, epilogue warp)
  int T;
  int* status;          // status word of the call (workspace)
  int zero_status;      // this launch is the first of its call: its first thread clears the status word
  int dependent;        // host side: launch as a programmatic dependent of the kernel before it in the stream
  int sub_stages;       // chained epilogues: K stages per accumulator hand-off (<= seg_stages; chains of fp32 tensor mode)
  int* sticky;          // this device's slot of the host-visible status array, or null
  uint32_t idesc;
  // split-K (store epilogues): work units [0, units_full) are whole tiles; each later tile is cut into
  // `split` K-stage ranges whose fp32 accumulators are parked in split_ws[slot][BM][BN]; the fix-up
  // kernel adds the parts in index order, adds the noise and stores the tile.  Nobody waits.
  // (Tried: the part that finishes last -- a ticket per tile -- sums the parts inside this kernel.
  // At B=16, T=1024, 1024->3072 that took 0.19 ms against 0.10 ms with the separate launch: the
  // sums then sit on the critical path of a few warps instead of spreading over the whole GPU.)
  int units_full, split;
  int park_whole;       // host side: the tiles from units_full on are parked even with split = 1
  // store GEMMs without a K split: the tiles from units_full on are cut into `cut` column parts (1 or 2)
  int cut;
  float* split_ws;
  // EPI_STORE_SCALED: K is `segs` segments (samples; 0: the factors are in the operand, one segment) of
  // `seg_stages` stages; every segment has its own
  // accumulator, scaled by that sample's clip factor when it is drained.  The factors come either from
  // `factors` (global, computed by an earlier kernel) or, when norm_partials != null, from the norm
  // pass's partial sums: the epilogue warps reduce them into shared memory while the first main loop
  // runs, and the first CTA also writes the norms and factors out.
  const float* factors;
  int segs, seg_stages;
  const float* norm_partials; int norm_nparts; float C, clamp;
  float* norms_ws; float* factors_ws; float* norms_out; float* factors_out;
  // EPI_GRAM: the T x T plane of a sample is cut into 128 x 128 blocks; only blocks (i, j) with j >= i
  // are computed (weight 2, the diagonal ones weight 1).  A work unit is one t-block i against TWO
  // s-blocks j1, j2 (an N = 256 MMA whose B stage is filled by two 128-row copies), see gram_decode;
  // at most one unit per sample has a single block (N = 128, idesc_half).  Units are numbered sample
  // by sample and all cost the same, so round-robin dealing is balanced.
  int gram_nb;          // 128-row blocks per sample
  uint32_t idesc_half;
  // store epilogue: optional bias[N] (same 16-bit type as the operands) added to every row
  const void* bias; int bias_dt; int bias_vec;   // bias_vec: 16-byte aligned
  // fp32 inputs as three bf16 products (EPI_SPLIT_*).  Both operand matrices are then [rows, 2n]: the high
  // bf16 halves of the n columns, then the low halves (x = hi + lo up to 2^-18 |x|); plane_a / plane_b is the
  // column offset of the low halves.  A K stage holds all four tiles -- A hi, A lo, B hi, B lo -- and feeds
  // three products, hi*lo, lo*hi and hi*hi, into the same accumulator (lo*lo, 2^-18 of the product, is
  // dropped): four tile loads for three products instead of six.  EPI_SPLIT6_*: [rows, 3n], x = hi + mid + lo
  // up to 2^-27 |x|, and the six products down to 2^-18 (what is dropped is below 2^-26): fp32 accuracy.
  int plane_a, plane_b;
  // store GEMMs: tiles are walked in groups of m_group tile rows (0 = plain order), so that the CTAs
  // running together cover a squarer patch of the output and re-read less of the operands
  int m_group;
  // the output cannot be written by the copy engine (row pitch or base not a multiple of 16 bytes)
  int direct_out;
  int flush_stages;     // with `keep`: a sample's sum goes to the kept tile every so many K stages (0: at its end), keep_add32
  float* keep;          // chained EPI_*_SUMSQ (may be null): the product tiles, [tile][CTA of the pair][box]
};

// ---- PTX wrappers (mbarrier helpers live in fdp_async.cuh) --------------------------------------------
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
// ---- CTA-pair (cta_group::2) helpers: the even CTA of a 2-CTA cluster issues one 256-row MMA for both;
// loads are per CTA (no multicast), completion is signalled on the leader's mbarrier ------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Hands an accumulator back to the leader's MMA warp.  Relaxed: no memory is handed over with it, the accumulator's loads
// have completed (tcgen05.wait::ld), and tcgen05.fence::before_thread_sync here and ::after_thread_sync behind the MMA warp's
// wait order them before its MMAs, for which the PTX manual's patterns between threads use a relaxed arrive and wait too.  A release at cluster scope waits for the warp's
// own earlier stores and took 1300 to 2500 cycles, in which the pair's tensor cores ran dry (weight gradients in six products,
// 16 x 197 rows 768 -> 3072: 151 us, now 134; 5 x 704, 64 -> 7928: 153 / 121; one pair alone in three products, 8192 deep: 89 / 64).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(leader_bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(leader_bar) : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair.  (One commit to both, not one each: a commit holds
// the tensor pipe up by about 30 cycles; 32768 rows 4096 -> 4096 bf16: 732 -> 699 us.)
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t r[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// shared-memory matrix descriptor (sm_100 format): start address, leading / stride byte offsets in
// 16-byte units, version 1, 128-byte swizzle.  The low word holds the address (and the leading offset), so that what
// moves with the stage and the K slice is one 32-bit addition.
struct Desc { uint32_t lo, hi; };
__device__ __forceinline__ Desc make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  Desc d;
  d.lo = ((saddr >> 4) & 0x3FFF) | (((lbo_bytes >> 4) & 0x3FFF) << 16);
  d.hi = ((sbo_bytes >> 4) & 0x3FFF) | (1u << 14) /* descriptor version of sm_100 */ | (2u << 29) /* SWIZZLE_128B */;
  return d;
}
// Descriptor of an operand whose first stage is at `saddr`, and the step of its low word to the k16-th UMMA_K slice.
//  MN-major: 64-element (128 B) MN chunks of BK rows each, chunk stride BK*128 B (leading offset),
//            8-row groups 1024 B apart (stride offset); a K=16 slice is 16 rows = 2048 B further.
//  K-major : rows of 128 B (64 K elements), 8-row groups 1024 B apart; a K=16 slice is 32 B further.
template <bool MN_MAJOR>
__device__ __forceinline__ Desc operand_desc(uint32_t saddr) { return make_desc(saddr, MN_MAJOR ? BK * 128 : 0, 1024); }
template <bool MN_MAJOR>
__device__ __forceinline__ constexpr uint32_t slice_step(int k16) { return (k16 * UMMA_K * (MN_MAJOR ? 128 : 2)) >> 4; }
template <int CTAS>
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 a, {%1, %2};\n\t"
      "mov.b64 b, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::%7.kind::f16 [%0], a, b, %5, p;\n\t}"
      ::"r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "n"(CTAS) : "memory");
}
// one lane of the warp, the same one every time
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}

// The Gaussian noise of 32 adjacent output elements starting at flat index idx0 (a multiple of 4: the
// tensor-core kernels only see row pitches and column offsets that are multiples of 8).
__device__ __forceinline__ void add_noise32(const NoiseKey& nk, size_t idx0, float v[32]) {
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    float z[4];
    noise_group(nk, (idx0 >> 2) + g, z);
    v[4 * g] += z[0]; v[4 * g + 1] += z[1]; v[4 * g + 2] += z[2]; v[4 * g + 3] += z[3];
  }
}

// v[0..31] += bias[n .. n+31]; the same address in every lane.  16-byte loads: the columns are few, the
// loads many (one set per 32 accumulator columns and warp), and as 32 scalar loads with a type switch
// each they took half of the forward GEMM's time at K = 1024.
__device__ __forceinline__ void add_bias32(const TcArgs& args, int n, float v[32]) {
  if (args.bias_vec && n + 32 <= args.N) {
    if (args.bias_dt == FDP_F32) {
      const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(args.bias) + n);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 b = __ldg(p + j);
        v[4 * j] += b.x; v[4 * j + 1] += b.y; v[4 * j + 2] += b.z; v[4 * j + 3] += b.w;
      }
    } else {
      const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(args.bias) + n);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 raw = __ldg(p + j);
        float b[8];
        if (args.bias_dt == FDP_BF16) unpack16<__nv_bfloat16>(raw, b); else unpack16<__half>(raw, b);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[8 * j + e] += b[e];
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (n + j < args.N) v[j] += load_as(args.bias, args.bias_dt, n + j);
  }
}

// ---- output boxes ------------------------------------------------------------------------------------
// After tcgen05.ld a lane holds one row of the tile, so direct stores put the 32 lanes of an instruction
// on 32 different rows: half-used sectors, 32 lines per request (16384 rows, 1024 -> 3072, bf16 forward with
// bias: 171 us, tensor pipe 27 % busy; 86 us with the boxes and add_bias32).  Instead every epilogue warp
// writes boxes of 32 rows x 128 bytes into its own 4 KB of shared memory, in the 128-byte swizzle of the
// tensor map (16-byte chunk j of row r at slot j ^ (r & 7): no bank conflicts), and one lane hands each box
// to the copy engine, which also clips what lies past the matrix.
__device__ __forceinline__ void box_wait(int lane) {      // the previous box has been read out
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ void box_put(uint32_t box, int lane, int j, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
               ::"r"(box + lane * 128 + ((j ^ (lane & 7)) << 4)), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void box_send(uint32_t box, const CUtensorMap* map, int col, int row, int lane) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(col), "r"(row), "r"(box) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
}
__device__ __forceinline__ void box_drain(int lane) {     // before the CTA leaves
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// 32 fp32 values per lane = one box
__device__ __forceinline__ void store_f32x32(uint32_t box, const CUtensorMap* map, const float v[32], int col, int row, int lane) {
  box_wait(lane);
#pragma unroll
  for (int j = 0; j < 8; ++j)
    box_put(box, lane, j, __float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]), __float_as_uint(v[4 * j + 2]),
            __float_as_uint(v[4 * j + 3]));
  box_send(box, map, col, row, lane);
}
// A kept product leaves straight from the registers, 32 x 32 elements at a time in the order that suits them: element
// group j (four columns) of all 32 rows, then the next, so that every store of a warp is 512 contiguous bytes.  Through
// shared memory and the copy engine, as an output goes, the stores compete with the operands for shared memory
// (16 x 512 rows, 4096 -> 4096 bf16: 336 us with tensor stores, 298 with whole boxes, 273 so).  weighted_sum_kernel knows the order.
__device__ __forceinline__ void keep_f32x32(float* dst, const float v[32], int lane) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    reinterpret_cast<float4*>(dst)[j * 32 + lane] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}
// A long sample's sum in two levels: what has been summed since the last time goes to the kept tile, or is added to what this
// lane left there, and the registers start again.
__device__ __forceinline__ void keep_add32(float* dst, float v[32], int lane, bool first, bool last) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float4* q = reinterpret_cast<float4*>(dst) + j * 32 + lane;
    if (!first) {
      const float4 x = *q;
      v[4 * j] += x.x; v[4 * j + 1] += x.y; v[4 * j + 2] += x.z; v[4 * j + 3] += x.w;
    }
    if (!last) {
      *q = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      v[4 * j] = 0.f; v[4 * j + 1] = 0.f; v[4 * j + 2] = 0.f; v[4 * j + 3] = 0.f;
    }
  }
}
// chunk c4 (32 columns) of a warp's 128 columns, in the output type; 16-bit types fill a box with two chunks
__device__ __forceinline__ void store_out32(const TcArgs& args, uint32_t box, const CUtensorMap* map, const float v[32], int c4,
                                            int col0, int row, int lane) {
  if (args.out_dt == FDP_F32) {
    if (col0 + 32 * c4 < args.N) store_f32x32(box, map, v, col0 + 32 * c4, row, lane);
    return;
  }
  if (col0 + 64 * (c4 >> 1) >= args.N) return;
  if ((c4 & 1) == 0) box_wait(lane);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint4 w;
    if (args.out_dt == FDP_BF16) w = pack16<__nv_bfloat16>(v + 8 * j); else w = pack16<__half>(v + 8 * j);
    box_put(box, lane, 4 * (c4 & 1) + j, w.x, w.y, w.z, w.w);
  }
  if ((c4 & 1) == 1) box_send(box, map, col0 + 64 * (c4 >> 1), row, lane);
}

// An epilogue warp's columns of an output that the copy engine cannot write: 32 at a time through the box all the same,
// then row by row, so that an instruction writes 32 adjacent elements; eight rows at a time, or each row would wait for its
// own trip through shared memory (16960 rows 79 -> 5597 fp32 229 us one by one, 175 now; 65502 rows 208 -> 494 fp16 95 / 60).  The noise
// is drawn per element here: a row pitch that is no multiple of four puts an element group across rows.  All of this is
// one loop, whose only part that depends on the registers' numbers is the filling of the box: unrolled over columns, types
// and rows it held 96 copies of the noise generator, and a warp that skipped them waited for instructions all the way
// (weight gradient of 39 x 21 rows, 5730 -> 1152 fp32, without noise 538 us, now 472, with it 773 / 555; 2 x 5, 642 -> 296 bf16 43 / 16).
__device__ __forceinline__ void box_fill(uint32_t box, const float v[32], int lane) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    box_put(box, lane, j, __float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]), __float_as_uint(v[4 * j + 2]),
            __float_as_uint(v[4 * j + 3]));
}
__device__ __forceinline__ float box_at(uint32_t box, int r, int lane) {
  float x;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(box + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4) : "memory");
  return x;
}
template <typename T>
__device__ __forceinline__ void store_box_rows(T* out, size_t ld, uint32_t box, int rows, int lane, bool in) {
#pragma unroll 1
  for (int r0 = 0; r0 < rows; r0 += 8, out += 8 * ld) {
    float x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = box_at(box, r0 + k, lane);      // (the box holds 32 rows, whatever the matrix has)
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (in && r0 + k < rows) out[k * ld] = from_f32<T>(x[k]);
  }
}
__device__ __forceinline__ void store_rows(const TcArgs& args, uint32_t box, const float v[128], int chunks, int n0, int row,
                                           int lane, bool noise) {
  const int rows = min(BOX_ROWS, args.M - row);
  const size_t ld = static_cast<size_t>(args.ld_out);
#pragma unroll 1
  for (int c4 = 0; c4 < chunks && n0 + c4 * 32 < args.N; ++c4) {
    box_wait(lane);       // a parked part may still be on its way out of the box
    switch (c4) {
      case 0: box_fill(box, v, lane); break;
      case 1: box_fill(box, v + 32, lane); break;
      case 2: box_fill(box, v + 64, lane); break;
      default: box_fill(box, v + 96, lane); break;
    }
    __syncwarp();
    const int n = n0 + c4 * 32 + lane;
    const bool in = n < args.N;
    const size_t idx = static_cast<size_t>(row) * ld + n;
    if (noise) {
#pragma unroll 2
      for (int r = 0; r < rows; ++r)
        if (in) store_as(args.out, args.out_dt, idx + r * ld, box_at(box, r, lane) + noise_at(args.nk, idx + r * ld));
    } else if (args.out_dt == FDP_F32) {
      store_box_rows(static_cast<float*>(args.out) + idx, ld, box, rows, lane, in);
    } else if (args.out_dt == FDP_BF16) {
      store_box_rows(static_cast<__nv_bfloat16*>(args.out) + idx, ld, box, rows, lane, in);
    } else {
      store_box_rows(static_cast<__half*>(args.out) + idx, ld, box, rows, lane, in);
    }
    __syncwarp();         // the box may be filled again
  }
}

// accr[4g .. 4g+3] += z * f with g known only at run time: a switch keeps every index static, so
// the 128 accumulators stay in registers.
__device__ __forceinline__ void add_group(float (&accr)[128], int g, const float z[4], float f) {
#define FDP_ADD_GROUP(G) case G: accr[4 * G] = fmaf(z[0], f, accr[4 * G]); accr[4 * G + 1] = fmaf(z[1], f, accr[4 * G + 1]); \
    accr[4 * G + 2] = fmaf(z[2], f, accr[4 * G + 2]); accr[4 * G + 3] = fmaf(z[3], f, accr[4 * G + 3]); break;
  switch (g) {
    FDP_ADD_GROUP(0) FDP_ADD_GROUP(1) FDP_ADD_GROUP(2) FDP_ADD_GROUP(3) FDP_ADD_GROUP(4) FDP_ADD_GROUP(5)
    FDP_ADD_GROUP(6) FDP_ADD_GROUP(7) FDP_ADD_GROUP(8) FDP_ADD_GROUP(9) FDP_ADD_GROUP(10) FDP_ADD_GROUP(11)
    FDP_ADD_GROUP(12) FDP_ADD_GROUP(13) FDP_ADD_GROUP(14) FDP_ADD_GROUP(15) FDP_ADD_GROUP(16) FDP_ADD_GROUP(17)
    FDP_ADD_GROUP(18) FDP_ADD_GROUP(19) FDP_ADD_GROUP(20) FDP_ADD_GROUP(21) FDP_ADD_GROUP(22) FDP_ADD_GROUP(23)
    FDP_ADD_GROUP(24) FDP_ADD_GROUP(25) FDP_ADD_GROUP(26) FDP_ADD_GROUP(27) FDP_ADD_GROUP(28) FDP_ADD_GROUP(29)
    FDP_ADD_GROUP(30) FDP_ADD_GROUP(31)
    default: break;
  }
#undef FDP_ADD_GROUP
}

// ---- the kernel ---------------------------------------------------------------------------------------
// CTAS = 2: a cluster of two CTAs works on one 256x256 tile.  Each CTA loads its 128 rows of A and
// its 128 columns of B (32 KiB per stage instead of 48, six stages), the even CTA issues
// tcgen05.mma.cta_group::2 (M = 256) for both, each CTA drains its own 128 accumulator rows.
template <bool A_MN, bool B_MN, int EPI, int CTAS>
__global__ void __launch_bounds__(threads_for(EPI), 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2,
               const __grid_constant__ CUtensorMap tmOut, const __grid_constant__ TcArgs args) {
  constexpr int PLANES = epi_planes(EPI);                // bf16 parts of fp32 operands
  constexpr int NST = ((CTAS == 2) ? 6 : STAGES) / PLANES;   // ring depth
  constexpr int A_BYTES = PLANES * A_STAGE_BYTES;
  constexpr int B_BYTES = B_STAGE_BYTES / CTAS;          // this CTA's share of (one half of) the B stage
  constexpr int STG = A_BYTES + PLANES * B_BYTES;
  constexpr int BN_CTA = BN / CTAS;                      // B columns (rows if K-major) loaded by this CTA
  constexpr int EPI_WARPS = epi_warps_for(EPI);
  constexpr bool CUTS = epi_plain(EPI);                  // may have units of half a tile's columns
  static_assert(NST * STG <= STAGES * STAGE_BYTES, "ring size");
  static_assert(CTAS == 1 || EPI_WARPS == 8, "pairs: eight epilogue warps");
  const uint32_t cta_rank = (CTAS == 2) ? cluster_ctarank() : 0u;
  const bool is_leader = cta_rank == 0;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* gen_base = smem_raw + (base - raw_addr);
  // ring | output boxes of the epilogue warps (store epilogues) | barriers | clip factors
  constexpr int BOXES = epi_stores(EPI) ? EPI_WARPS * BOX_BYTES : 0;
  const uint32_t bar_base = base + NST * STG + BOXES;
  uint8_t* bar_gen = gen_base + NST * STG + BOXES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (NST + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * NST + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * NST + 2 + a); };
  const uint32_t drain_bar = bar_base + 8u * (2 * NST + 4);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_gen + 8 * (2 * NST + 5));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_gen + 8 * (2 * NST + 5) + 4);
  float* sfac = reinterpret_cast<float*>(bar_gen + BAR_BYTES);   // EPI_STORE_SCALED: clip factors [segs]
  const WaitCtx wctx{abort_flag, args.status, args.sticky, WAIT_LIMIT_CYCLES};

  constexpr int NUM_ACC = (EPI == EPI_GRAM) ? 1 : 2;
  // six products: accumulator hand-offs per K stage.  In the norm pass the truncation of the accumulators does not
  // average out over the elements (it shrinks all of them), so its chains hold two large steps instead of four.
  constexpr int SUBS = (EPI == EPI_SPLIT6_SUMSQ) ? 2 : 1;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform, and known to be)
  const int total_tiles = args.batch * args.tiles_per_batch;
  const int kst_total = args.k_stages + (EPI == EPI_GRAM ? args.k_stages2 : 0);
  const int total_units = args.units_full + (total_tiles - args.units_full) * args.split * (CUTS ? args.cut : 1);

  if (threadIdx.x == 0) {
    // (a wait can only run out a second from now, so no report of this call can precede the clearing)
    if (args.zero_status && blockIdx.x == 0 && args.status != nullptr) *args.status = 0;
    for (int s = 0; s < NST; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), EPI_WARPS * CTAS); }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (CTAS == 2) {
    // the peer's barriers must be initialised before anything is signalled across the pair
    __syncthreads();
    cluster_sync_all();
  }
  if (warp == 1) {
    if (CTAS == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                   ::"r"(smem_u32(const_cast<uint32_t*>(tmem_slot))), "r"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                   ::"r"(smem_u32(const_cast<uint32_t*>(tmem_slot))), "r"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Barriers, TMEM and the shared-memory carve-up are ready.  Let the kernel that follows in the
  // stream be scheduled as SMs free up (it waits at this same point), and, if this launch is itself
  // a programmatic dependent, wait here for the kernel before it: nothing above touched global
  // memory that an earlier kernel writes.
  pdl_trigger();
  pdl_wait();
  // work is dealt to CTAs (or CTA pairs) round-robin
  const int wid = blockIdx.x / CTAS, wstep = gridDim.x / CTAS;
  const uint32_t tmem_base = *tmem_slot;

  // tile -> (batch, m0, n0, half).  EPI_GRAM: m0 = first row of the t-block, n0 / n1 = first rows of
  // the two s-blocks (n1 < 0 and half = 1 for a single-block unit)
  int gram_n1 = -1;
  auto decode = [&](int tile, int& b, int& m0, int& n0, int& half) {
    half = 0;
    b = tile / args.tiles_per_batch;
    int q = tile - b * args.tiles_per_batch;
    if (EPI == EPI_GRAM) {
      int i, j1, j2;
      gram_decode(args.gram_nb, q, i, j1, j2);
      m0 = i * BM; n0 = j1 * BM;
      gram_n1 = j2 >= 0 ? j2 * BM : -1;
      half = j2 < 0;
      return;
    }
    int mi, ni;
    if (args.n_fastest) {
      ni = q % args.tiles_n; mi = q / args.tiles_n;
    } else if (args.m_group > 0) {
      const int per_group = args.m_group * args.tiles_n;
      const int g = q / per_group, r = q - g * per_group;
      const int gm = min(args.m_group, args.tiles_m - g * args.m_group);
      mi = g * args.m_group + r % gm; ni = r / gm;
    } else {
      mi = q % args.tiles_m; ni = q / args.tiles_m;
    }
    m0 = mi * (BM * CTAS) + cta_rank * BM;
    n0 = ni * BN;
  };

  // work unit -> tile, K-stage range, slot in split_ws (-1: whole tile, normal epilogue); a unit of half a tile's
  // columns is named by ncut: which half, -1 for a whole tile
  auto decode_unit = [&](int u, int& tile, int& ks0, int& ks1, int& slot, int& ncut) {
    ncut = -1;
    if (u < args.units_full) { tile = u; ks0 = 0; ks1 = kst_total; slot = -1; return; }
    const int v = u - args.units_full;
    if (CUTS && args.cut == 2) {
      tile = args.units_full + (v >> 1); ncut = v & 1; ks0 = 0; ks1 = kst_total; slot = -1;
      return;
    }
    const int part = v % args.split;
    tile = args.units_full + v / args.split;
    ks0 = static_cast<int>(static_cast<long long>(kst_total) * part / args.split);
    ks1 = static_cast<int>(static_cast<long long>(kst_total) * (part + 1) / args.split);
    slot = v;
  };
  // Chained epilogues hand an accumulator over every sub_stages stages, counted from the sample's start, and at the
  // sample's and the unit's end.  (With fp32 inputs it is a few stages only: the tensor cores add into the
  // TMEM accumulator by truncation, about one unit in the last place per K = 16 step and all of one sign, so a
  // long chain drifts; short chains summed in registers with round-to-nearest do not.)
  // running number of the hand-off that contains stage ks
  auto segment_index = [&](int ks) {
    const int sg = ks / args.seg_stages;
    return sg * ((args.seg_stages + args.sub_stages - 1) / args.sub_stages) + (ks - sg * args.seg_stages) / args.sub_stages;
  };

  if (warp == 0) {
    // ================= TMA producer (the warp walks the loop, one elected lane issues) =================
    {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int u = wid; u < total_units && ok; u += wstep) {
        int tile, ks0, ks1, slot, b, m0, n0, half, ncut;
        decode_unit(u, tile, ks0, ks1, slot, ncut);
        decode(tile, b, m0, n0, half);
        const bool narrow = CUTS && ncut >= 0;
        if (narrow) n0 += ncut * (BN / 2);
        const int row0 = b * args.batch_rows;
        // K range along the rows: sample z, row t of it.  The maps are three-dimensional (column, row of the
        // sample, sample), so the rows a sample's last stage is short of read as zeros, whatever its length.
        int z = 0, t = 0;
        if (A_MN && B_MN) { z = b + ks0 / args.seg_stages; t = ks0 % args.seg_stages * BK; }
        for (int ks = ks0; ks < ks1; ++ks) {
          if (!mbar_wait_warp(empty_bar(stage), phase ^ 1u, wctx, 1)) { ok = false; break; }
          const bool second = (EPI == EPI_GRAM) && ks >= args.k_stages;
          const CUtensorMap* ma = second ? &tmA2 : &tmA;
          const CUtensorMap* mb = second ? &tmB2 : &tmB;
          const int k0 = (second ? ks - args.k_stages : ks) * BK;
          const uint32_t sa = base + stage * STG, sb = sa + A_BYTES;
          if (elect_one()) {
          if (EPI == EPI_GRAM) {
            // A: the t-block; B: two independent 128-row s-blocks, one per half of the stage
            // (a unit that contains the diagonal block (i, i) has its t-block in the B stage already:
            // the MMA warp points the A descriptor there and no A copy is made)
            constexpr uint32_t HALF_B = B_STAGE_BYTES / 2;
            const bool a_in_b = (n0 == m0) || (gram_n1 == m0);
            mbar_expect_tx(full_bar(stage), (a_in_b ? 0 : A_STAGE_BYTES) + (gram_n1 >= 0 ? 2 : 1) * HALF_B);
            if (!a_in_b) tma_load_2d(sa, ma, k0, row0 + m0, full_bar(stage));
            tma_load_2d(sb, mb, k0, row0 + n0, full_bar(stage));
            if (gram_n1 >= 0) tma_load_2d(sb + HALF_B, mb, k0, row0 + gram_n1, full_bar(stage));
          } else {
            // both CTAs' copies of a pair complete on the leader's barrier, which expects the bytes of both
            const uint32_t lbar = CTAS == 1 ? full_bar(stage) : mapa_u32(full_bar(stage), 0);
            if (is_leader) mbar_expect_tx(full_bar(stage), CTAS * (narrow ? A_BYTES + PLANES * B_BYTES / 2 : STG));
            const int nb0 = n0 + static_cast<int>(cta_rank) * (narrow ? BN_CTA / 2 : BN_CTA);
            auto load = [&](uint32_t dst, const CUtensorMap* map, int c0, int c1) {
              if (CTAS == 1) tma_load_2d(dst, map, c0, c1, lbar); else tma_load_2d_pair(dst, map, c0, c1, lbar);
            };
            auto load3 = [&](uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2) {
              if (CTAS == 1) tma_load_3d(dst, map, c0, c1, c2, lbar); else tma_load_3d_pair(dst, map, c0, c1, c2, lbar);
            };
#pragma unroll
            for (int pl = 0; pl < PLANES; ++pl) {
              const int ca = pl * args.plane_a, cb = pl * args.plane_b;
              const uint32_t da = sa + pl * A_STAGE_BYTES, db = sb + pl * B_BYTES;
              if (A_MN) {
#pragma unroll
                for (int i = 0; i < BM / 64; ++i) load3(da + i * (BK * 128), ma, m0 + 64 * i + ca, t, z);
              } else if (EPI == EPI_SPLIT6_STORE) {     // (column, part, row): a K stage that ends past the last column reads zeros
                load3(da, ma, k0, pl, m0);
              } else {
                load(da, ma, k0 + ca, m0);
              }
              if (B_MN) {
#pragma unroll
                for (int j = 0; j < BN_CTA / 64; ++j) {
                  if (narrow && j >= BN_CTA / 128) break;
                  if (A_MN) load3(db + j * (BK * 128), mb, nb0 + 64 * j + cb, t, z);
                  else if (EPI == EPI_SPLIT6_STORE) load3(db + j * (BK * 128), mb, nb0 + 64 * j, pl, k0);
                  else load(db + j * (BK * 128), mb, nb0 + 64 * j + cb, k0);
                }
              } else if (EPI == EPI_SPLIT6_STORE) {
                load3(db, narrow ? &tmB2 : mb, k0, pl, nb0);
              } else {
                load(db, narrow ? &tmB2 : mb, k0 + cb, nb0);    // tmB2: boxes of half the rows
              }
            }
          }
          }
          __syncwarp();
          if (A_MN && B_MN) {
            t += BK;
            if (t >= args.seg_stages * BK) { t = 0; ++z; }
          }
          if (++stage == NST) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok && lane == 0) {
        // wait (bounded) for the copies already in flight before the CTA may leave
        for (int s = 0; s < NST; ++s) {
          const long long t0 = clock64();
          const uint32_t ph = (s < stage) ? phase : (phase ^ 1u);
          while (!mbar_try(full_bar(s), ph) && clock64() - t0 < WAIT_LIMIT_CYCLES / 8) {}
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (the leader CTA of a pair issues for both) =================
    // The whole warp walks the loop and one elected lane issues, so that addresses and descriptors stay in uniform
    // registers: issued from a branch of one lane, an instruction took about 130 cycles, as long as the 256 x 256 x 16
    // product itself, and every wait of the loop held the tensor cores up (one pair alone, 256 x 256 tile: 0.30 us a K stage
    // whatever the ring's depth, now 0.19; 16384 rows, 1024 -> 3072 bf16: 83 us, now 74; 32768 x 4096 x 4096 clipped sum
    // with its norms 1007 -> 897).
    auto commit = [&](uint32_t bar) {   // signals `bar` (in both CTAs of a pair) when the MMAs issued so far are done
      if (CTAS == 1) tc_commit(bar); else tc_commit_pair(bar);
    };
    if (is_leader) {
      int stage = 0; uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      const Desc a0 = operand_desc<A_MN>(base), b0 = operand_desc<B_MN>(base + A_BYTES);
      // products of a K slice, by the parts of A and B they take.  Three: hi*lo, lo*hi, hi*hi.  Six, smallest first (the
      // accumulator is added to by truncation, one unit in its last place per step, so the steps that come before it is
      // large cost nothing): hi*lo, lo*hi, mid*mid, hi*mid, mid*hi, hi*hi.
      constexpr int PRODUCTS = PLANES == 3 ? 6 : PLANES == 2 ? 3 : 1;
      constexpr int PA[3][6] = {{0}, {0, 1, 0}, {0, 2, 1, 0, 1, 0}}, PB[3][6] = {{0}, {1, 0, 0}, {2, 0, 1, 1, 0, 0}};
      // issues the products of K slices [k0, k1) of the stage at offset `so`, in slices or product by product
      auto issue = [&](uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, auto k0, auto k1, bool fresh) {
        auto one = [&](int q, int k16, bool first) {
          tc_mma<CTAS>(d, a_lo + PA[PLANES - 1][q] * (A_STAGE_BYTES >> 4) + slice_step<A_MN>(k16), a0.hi,
                       b_lo + PB[PLANES - 1][q] * (B_BYTES >> 4) + slice_step<B_MN>(k16), b0.hi, idesc, first && fresh ? 0u : 1u);
        };
        if constexpr (PLANES == 3) {
#pragma unroll
          for (int q = 0; q < PRODUCTS; ++q)
#pragma unroll
            for (int k16 = k0; k16 < k1; ++k16) one(q, k16, q == 0 && k16 == k0);
        } else {
#pragma unroll
          for (int k16 = k0; k16 < k1; ++k16)
#pragma unroll
            for (int q = 0; q < PRODUCTS; ++q) one(q, k16, q == 0 && k16 == k0);
        }
      };
      for (int u = wid; u < total_units && ok; u += wstep) {
        int tile, ks0, ks1, slot, tb, tm0, tn0, half, ncut;
        decode_unit(u, tile, ks0, ks1, slot, ncut);
        decode(tile, tb, tm0, tn0, half);
        // a single-block unit multiplies by the first 128 rows of the B stage only (N = 128), half a tile likewise
        const uint32_t idesc = half || (CUTS && ncut >= 0) ? args.idesc_half : args.idesc;
        int ks = ks0;
        // stages left of the sample at ks, and how far into a hand-off a K split has put the unit's start
        int sample_left = 0, sub_off = 0;
        if (epi_chained(EPI)) {
          sample_left = args.seg_stages - ks0 % args.seg_stages;
          sub_off = (args.seg_stages - sample_left) % args.sub_stages;
        }
        // one accumulator per segment: the whole unit, or one sample's share of it for EPI_STORE_SCALED
        if constexpr (SUBS > 1) {
          for (; ks < ks1 && ok; ++ks) {
            if (!mbar_wait_warp(full_bar(stage), phase, wctx, 3)) { ok = false; break; }
            const uint32_t so = static_cast<uint32_t>(stage * STG) >> 4;
#pragma unroll
            for (int sub = 0; sub < SUBS; ++sub, ++it) {
              const int acc = it % NUM_ACC;
              if (!mbar_wait_warp(tempty_bar(acc), ((it / NUM_ACC) & 1u) ^ 1u, wctx, 2)) { ok = false; break; }
              tc_fence_after();
              if (elect_one()) {
                issue(tmem_base + acc * BN, a0.lo + so, b0.lo + so, idesc, sub * (4 / SUBS), (sub + 1) * (4 / SUBS), true);
                commit(tfull_bar(acc));
                if (sub == SUBS - 1) commit(empty_bar(stage));
              }
              __syncwarp();
            }
            if (!ok) break;
            if (++stage == NST) { stage = 0; phase ^= 1u; }
          }
        }
        while (ks < ks1 && ok) {
          const int seg_begin = ks;
          int seg_end = ks1;
          if (epi_chained(EPI)) {
            const int len = min(args.sub_stages - sub_off, sample_left);
            sub_off = 0;
            seg_end = min(ks + len, ks1);
            sample_left -= len;
            if (sample_left == 0) sample_left = args.seg_stages;
          }
          const int acc = it % NUM_ACC;
          const uint32_t acc_phase = (it / NUM_ACC) & 1u;
          if (!mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u, wctx, 2)) { ok = false; break; }
          tc_fence_after();
          for (; ks < seg_end; ++ks) {
            if (!mbar_wait_warp(full_bar(stage), phase, wctx, 3)) { ok = false; break; }
            tc_fence_after();
            const bool second = (EPI == EPI_GRAM) && ks >= args.k_stages;
            const uint32_t d = tmem_base + (EPI == EPI_GRAM ? (second ? BN : 0) : acc * BN);
            const bool first_stage = second ? (ks == args.k_stages) : (ks == seg_begin);
            const uint32_t so = static_cast<uint32_t>(stage * STG) >> 4;
            uint32_t a_lo = a0.lo + so;
            const uint32_t b_lo = b0.lo + so;
            if (EPI == EPI_GRAM) {   // diagonal block in this unit: A is the matching half of the B stage
              if (tn0 == tm0) a_lo = b_lo;
              else if (gram_n1 == tm0) a_lo = b_lo + (B_STAGE_BYTES / 2 >> 4);
            }
            if (elect_one()) {
              issue(d, a_lo, b_lo, idesc, 0, BK / UMMA_K, first_stage);
              // frees the stage (in both CTAs of a pair) once these MMAs have read it
              commit(empty_bar(stage));
              if (ks + 1 == seg_end) commit(tfull_bar(acc));
            }
            __syncwarp();
            if (++stage == NST) { stage = 0; phase ^= 1u; }
          }
          if (ok) ++it;
        }
      }
      if (!ok && elect_one()) {
        // let MMAs already issued finish before TMEM is released
        commit(drain_bar);
        const long long t0 = clock64();
        while (!mbar_try(drain_bar, 0) && clock64() - t0 < WAIT_LIMIT_CYCLES / 8) {}
      }
    }
  } else {
    // ================= epilogue: warps 2.., TMEM lane quarter = warp % 4 =================
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int ew = warp - 2;
    const uint32_t box = base + NST * STG + ew * BOX_BYTES;
    // where box c4 of this warp's part of a kept tile goes
    auto kept_box = [&](int tile, int c4) {
      return args.keep + (((static_cast<size_t>(tile) * CTAS + cta_rank) * EPI_WARPS + ew) * 4 + c4) * 1024;
    };
    int it = 0;
    bool ok = true;
    if (epi_scaled(EPI) && args.norm_partials != nullptr) {
      // clip factors of all samples from the norm pass's partial sums (fixed order: a lane adds every
      // 32nd partial, then the shuffle tree), while the producer and MMA warps start the main loop
      for (int b = ew; b < args.segs; b += EPI_WARPS) {
        const float* pp = args.norm_partials + static_cast<size_t>(b) * args.norm_nparts;
        float sq = 0.f;
        for (int i = lane; i < args.norm_nparts; i += 32) sq += pp[i];
        sq = warp_sum(sq);
        if (lane == 0) {
          const float n = norm_of_sumsq(sq);
          const float f = clip_factor(n, args.C, args.clamp);
          sfac[b] = f;
          if (blockIdx.x == 0) {
            if (args.norms_out != nullptr) args.norms_out[b] = n;
            if (args.factors_out != nullptr) args.factors_out[b] = f;
          }
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");   // the eight epilogue warps
    }
    for (int u = wid; u < total_units && ok; u += wstep) {
      int tile, ks0, ks1, slot, b, m0, n0, half, ncut;
      decode_unit(u, tile, ks0, ks1, slot, ncut);
      decode(tile, b, m0, n0, half);
      const bool narrow = CUTS && ncut >= 0;
      if (narrow) n0 += ncut * (BN / 2);
      const int warp_cols = narrow ? BN / 4 : BN / 2;      // columns of an epilogue warp
      const int m = m0 + row;
      if constexpr (epi_chained(EPI)) {
        // eight warps: two per lane quarter, each owning 128 of the tile's 256 columns in registers
        const int chalf = ew >> 2;
        float accr[128];
#pragma unroll
        for (int i = 0; i < 128; ++i) accr[i] = 0.f;
        // A whole tile's Gaussian noise goes into the accumulators a few element groups per sample
        // segment, in the time these warps would otherwise wait for the next segment's MMAs; K-split
        // parts stay noise-free (the fix-up kernel adds the noise once per tile).
        const bool pre_noise = epi_scaled(EPI) && slot < 0 && args.nk.std != 0.f && m < args.M && !args.direct_out;
        const uint64_t g0 = (static_cast<uint64_t>(m) * args.ld_out + n0 + chalf * 128) >> 2;
        const int nseg = segment_index(ks1 - 1) - segment_index(ks0) + 1;
        // (no divisions from here on: what a hand-off takes between the commit and the arrival is time the tensor cores
        // wait when its MMAs are few)
        int ng = 0, noise_due = 0;
        int sample = ks0 / args.seg_stages, sample_left = (sample + 1) * args.seg_stages - ks0;
        int sub_off = (args.seg_stages - sample_left) % args.sub_stages;
        const int nb = n0 + chalf * 128;
        int flush_left = args.flush_stages;      // (0 never comes down to 0)
        bool flushed = false;
        for (int ks = ks0, sub = 0; ks < ks1 && ok; ++it) {
          const int acc = it % NUM_ACC;
          const uint32_t acc_phase = (it / NUM_ACC) & 1u;
          // the divisor goes into the factor, so the noise is added as it is drawn
          const float cbs = !epi_scaled(EPI) || args.segs == 0 ? args.scale
                          : (args.norm_partials != nullptr ? sfac[sample] : __ldg(args.factors + sample)) * args.scale;
          if (++sub == SUBS) {     // on to the next hand-off's first stage, as the MMA warp goes
            sub = 0;
            const int len = min(args.sub_stages - sub_off, sample_left);
            sub_off = 0;
            ks += len;
            sample_left -= len;
            if (sample_left == 0) { sample_left = args.seg_stages; ++sample; }
          }
          if (!mbar_wait_warp(tfull_bar(acc), acc_phase, wctx, 4)) { ok = false; break; }
          tc_fence_after();
          const uint32_t tb = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BN + chalf * warp_cols;
#pragma unroll
          for (int c4 = 0; c4 < 4; ++c4) {
            if (narrow && c4 >= 2) break;
            uint32_t r[32];
            tc_ld32(tb + c4 * 32, r);
            tc_wait_ld();
            if (c4 == 3 || (narrow && c4 == 1)) {     // the accumulator has been read: back to the MMA warp
              tc_fence_before();
              __syncwarp();
              if (lane == 0) {
                if (CTAS == 1 || is_leader) mbar_arrive(tempty_bar(acc));
                else mbar_arrive_cluster(mapa_u32(tempty_bar(acc), 0));
              }
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) accr[c4 * 32 + j] = fmaf(cbs, __uint_as_float(r[j]), accr[c4 * 32 + j]);
          }
          if constexpr (epi_planes(EPI) == 3 && epi_sumsq(EPI)) {
            if (sub == 0 && --flush_left == 0 && ks < ks1) {
              flush_left = args.flush_stages;
              if (m0 + quarter * 32 < args.M) {
#pragma unroll
                for (int c4 = 0; c4 < 4; ++c4)
                  if (nb + c4 * 32 < args.N) keep_add32(kept_box(tile, c4), accr + c4 * 32, lane, !flushed, false);
              }
              flushed = true;
            }
          }
          if (epi_scaled(EPI) && pre_noise) {
            for (noise_due += 32; noise_due >= nseg; noise_due -= nseg, ++ng) {
              float z[4];
              noise_group(args.nk, g0 + ng, z);
              add_group(accr, ng, z, 1.0f);
            }
          }
        }
        if (!ok) break;
        if constexpr (epi_sumsq(EPI)) {
          // the unit is one sample's product tile: its squares, without the rows and columns past the
          // matrix (with split operands a tile that overhangs reads the other half's columns, not zeros)
          float part = 0.f;
          if constexpr (epi_planes(EPI) == 3) {
            if (flushed && m0 + quarter * 32 < args.M) {
#pragma unroll
              for (int c4 = 0; c4 < 4; ++c4)
                if (nb + c4 * 32 < args.N) keep_add32(kept_box(tile, c4), accr + c4 * 32, lane, false, true);
            }
          }
          if (m < args.M) {
#pragma unroll
            for (int i = 0; i < 128; ++i) {
              const float a = (nb + i < args.N) ? accr[i] : 0.f;
              part = fmaf(a, a, part);
            }
          }
          part = warp_sum(part);
          if (lane == 0) args.partials[(static_cast<size_t>(tile) * CTAS + cta_rank) * EPI_WARPS + ew] = part;
          if (args.keep != nullptr && m0 + quarter * 32 < args.M) {
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4)
              if (nb + c4 * 32 < args.N) keep_f32x32(kept_box(tile, c4), accr + c4 * 32, lane);
          }
        } else if (slot < 0) {
          if (m0 + quarter * 32 < args.M) {
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
              if (narrow && c4 >= 2) break;
              const int n = n0 + chalf * warp_cols + c4 * 32;
              if (epi_plain(EPI) && args.bias != nullptr && n < args.N) add_bias32(args, n, accr + c4 * 32);
              if (EPI == EPI_SPLIT_STORE || !args.direct_out) store_out32(args, box, &tmOut, accr + c4 * 32, c4, n0 + chalf * warp_cols, m0 + quarter * 32, lane);
            }
            if (EPI != EPI_SPLIT_STORE && args.direct_out)       // (three products: rows and pointers of 16 bytes only)
              store_rows(args, box, accr, narrow ? 2 : 4, n0 + chalf * warp_cols, m0 + quarter * 32, lane, epi_scaled(EPI) && args.nk.std != 0.f);
          }
        } else {
          // park this part (already divided by the batch) for the fix-up kernel
#pragma unroll
          for (int c4 = 0; c4 < 4; ++c4)
            store_f32x32(box, &tmA2, accr + c4 * 32, chalf * 128 + c4 * 32, (slot * CTAS + cta_rank) * BM + quarter * 32, lane);
        }
        continue;
      }
      const int acc = it % NUM_ACC;
      const uint32_t acc_phase = (it / NUM_ACC) & 1u;
      if (!mbar_wait_warp(tfull_bar(acc), acc_phase, wctx, 4)) { ok = false; break; }
      tc_fence_after();
      const uint32_t tbase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + (EPI == EPI_GRAM ? 0 : acc * BN);
      float part = 0.f;
      if constexpr (EPI == EPI_STORE) {
        // this warp's 128 columns into registers, then the accumulator goes back to the MMA warp at once
        const int col0 = (ew >> 2) * warp_cols;
        float v[128];
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4) {
          if (narrow && c4 >= 2) break;
          tc_ld32(tbase + col0 + c4 * 32, reinterpret_cast<uint32_t*>(v) + c4 * 32);
        }
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CTAS == 1 || is_leader) mbar_arrive(tempty_bar(acc));
          else mbar_arrive_cluster(mapa_u32(tempty_bar(acc), 0));
        }
        ++it;
        if (slot >= 0) {   // K-split unit: park the raw accumulator for the fix-up kernel
#pragma unroll
          for (int c4 = 0; c4 < 4; ++c4)
            store_f32x32(box, &tmA2, v + c4 * 32, col0 + c4 * 32, (slot * CTAS + cta_rank) * BM + quarter * 32, lane);
        } else if (m0 + quarter * 32 < args.M) {
#pragma unroll
          for (int c4 = 0; c4 < 4; ++c4) {
            if (narrow && c4 >= 2) break;
            const int n = n0 + col0 + c4 * 32;
            float* w = v + c4 * 32;
#pragma unroll
            for (int j = 0; j < 32; ++j) w[j] *= args.scale;
            if (args.bias != nullptr && n < args.N) add_bias32(args, n, w);
            if (args.nk.std != 0.f && m < args.M && n < args.N)
              add_noise32(args.nk, static_cast<size_t>(m) * args.ld_out + n, w);
            if (!args.direct_out) store_out32(args, box, &tmOut, w, c4, n0 + col0, m0 + quarter * 32, lane);
          }
          if (args.direct_out) store_rows(args, box, v, narrow ? 2 : 4, n0 + col0, m0 + quarter * 32, lane, false);
        }
        continue;
      } else if (EPI == EPI_SUMSQ) {
        // rows / columns outside the matrix were zero-filled by TMA, so they add nothing
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t r[32];
          tc_ld32(tbase + c, r);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) { const float f = __uint_as_float(r[j]); part = fmaf(f, f, part); }
        }
      } else {
        // columns 0..127 belong to s-block n0, 128..255 to s-block gram_n1; a diagonal block counts
        // once, any other block twice (it stands for its mirror image too); rows and columns past the
        // end of the sample (they belong to the next one) count nothing
        const int t = m0 + row;
        const int ncols = half ? BN / 2 : BN;
#pragma unroll 1
        for (int c = 0; c < ncols; c += 32) {
          uint32_t p[32], q[32];
          tc_ld32(tbase + c, p);
          tc_ld32(tbase + BN + c, q);
          tc_wait_ld();
          const int sb0 = (c < BN / 2) ? n0 : gram_n1;          // first row of this chunk's s-block
          const int s0 = sb0 + (c & (BN / 2 - 1));
          const float wblk = (sb0 == m0) ? 1.f : 2.f;
          if (t < args.T) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float w = (s0 + j < args.T) ? wblk : 0.f;
              part = fmaf(w * __uint_as_float(p[j]), __uint_as_float(q[j]), part);
            }
          }
        }
      }
      // accumulator drained: hand it back to the MMA warp (of the leader CTA)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CTAS == 1 || is_leader) mbar_arrive(tempty_bar(acc));
        else mbar_arrive_cluster(mapa_u32(tempty_bar(acc), 0));
      }
      ++it;
      if (EPI == EPI_SUMSQ || EPI == EPI_GRAM) {
        // one partial per (unit, epilogue warp); units are numbered sample by sample
        part = warp_sum(part);
        if (lane == 0) args.partials[static_cast<size_t>(tile) * 4 + quarter] = part;
      }
    }
  }

  // ================= teardown =================
  if (epi_stores(EPI) && warp >= 2) box_drain(lane);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();  // neither CTA leaves (or frees TMEM) while its peer may still signal it
  if (warp == 1) {
    tc_fence_after();
    if (CTAS == 2)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---- split-K fix-up: out = scale * (part_0 + part_1 + ...) + noise for the K-split tiles --------------
__global__ void __launch_bounds__(256) splitk_fixup_kernel(const float* __restrict__ ws, int first_tile, int split,
                                                           int tile_rows, int M, int N, int tiles_m, int tiles_n, int n_fastest,
                                                           int m_group,
                                                           void* __restrict__ out, int out_dt, long long ld_out,
                                                           float scale, NoiseKey nk, const void* __restrict__ bias, int bias_dt) {
  pdl_wait();
  const int t = blockIdx.y;  // index among the split tiles
  const int q = first_tile + t;
  int mi, ni;  // the tile order of tc_gemm_kernel's decode
  if (n_fastest) {
    ni = q % tiles_n; mi = q / tiles_n;
  } else if (m_group > 0) {
    const int per_group = m_group * tiles_n;
    const int g = q / per_group, r = q - g * per_group;
    const int gm = min(m_group, tiles_m - g * m_group);
    mi = g * m_group + r % gm; ni = r / gm;
  } else {
    mi = q % tiles_m; ni = q / tiles_m;
  }
  const int m0 = mi * tile_rows, n0 = ni * BN;
  const int e = (blockIdx.x * 256 + threadIdx.x) * 4;  // element of the tile, 4 adjacent columns
  const int row = e / BN, col = e % BN;
  const int m = m0 + row, n = n0 + col;
  if (m >= M || n >= N) return;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int p = 0; p < split; ++p) {
    const float4 v = *reinterpret_cast<const float4*>(ws + (static_cast<size_t>(t * split + p) * tile_rows + row) * BN + col);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  float v[4] = {acc.x * scale, acc.y * scale, acc.z * scale, acc.w * scale};
  const size_t idx0 = static_cast<size_t>(m) * ld_out + n;
  if (bias != nullptr)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < N) v[j] += load_as(bias, bias_dt, n + j);
  if (nk.std != 0.f) {
    if ((idx0 & 3) == 0) {
      float z[4];
      noise_group(nk, idx0 >> 2, z);
      v[0] += z[0]; v[1] += z[1]; v[2] += z[2]; v[3] += z[3];
    } else {     // a row pitch that is no multiple of four
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] += noise_at(nk, idx0 + j);
    }
  }
  for (int j = 0; j < 4; ++j)
    if (n + j < N) store_as(out, out_dt, idx0 + j, v[j]);
}

// ---- the clipped sum of kept products: out = sum_b (c_b scale) P_b + noise ----------------------------------------
// HBM-bound: B fp32 tiles read once, one written.  A block takes one 32 x 32 box of every sample as an epilogue warp
// left it (keep_f32x32): four adjacent elements a thread, eight samples' loads under way, and the sum goes through
// shared memory so that rows are written in whole.  Eight samples are summed
// among themselves and then added to the rest, so the chain of the sum is an eighth of B.  WIDE, for six products: the sum
// runs in 64 bits, a chain in fp32 adds as much to the error of such a gradient as its products have, with the next four samples' loads
// under way (16 samples, 768 x 3072: 24.8 us in fp32, 27.9 so; 100 samples, 128 x 200: 33 / 26).
template <bool WIDE>
__global__ void __launch_bounds__(256, WIDE ? 4 : 6) weighted_sum_kernel(const float* __restrict__ P, const TcFactorSource fs, int B, int ctas,
                                                           int tiles_m, size_t sample_stride, int M, int N,
                                                           void* __restrict__ out, int out_dt, int vec_out, float scale, NoiseKey nk) {
  // box -> tile, CTA of the pair, epilogue warp (lane quarter, column half), 32 columns
  const int c4 = blockIdx.x & 3, ew = (blockIdx.x >> 2) & 7, rank = ctas == 2 ? (blockIdx.x >> 5) & 1 : 0;
  const int tile = blockIdx.x / (32 * ctas);
  const int mi = tile % tiles_m, ni = tile / tiles_m;
  const int m0 = (mi * ctas + rank) * BM + ((ew + 2) & 3) * 32, n0 = ni * BN + (ew >> 2) * 128 + c4 * 32;
  if (m0 >= M || n0 >= N) return;
  __shared__ float4 box[8][33];
  __shared__ float sfac[KEEP_SMEM_FACTORS];
  pdl_wait();
  if (fs.factors == nullptr) {     // few partials: every block derives the factors, as the per-sample epilogue does
    for (int b = threadIdx.x >> 5; b < B; b += 8) {
      const float* pp = fs.norm_partials + static_cast<size_t>(b) * fs.nparts;
      float sq = 0.f;
      for (int i = threadIdx.x & 31; i < fs.nparts; i += 32) sq += pp[i];
      sq = warp_sum(sq);
      if ((threadIdx.x & 31) == 0) {
        const float n = norm_of_sumsq(sq), f = clip_factor(n, fs.C, fs.clamp);
        sfac[b] = f;
        if (blockIdx.x == 8) {     // the box at row 0 and column 0, which every matrix has
          if (fs.norms_out != nullptr) fs.norms_out[b] = n;
          if (fs.factors_out != nullptr) fs.factors_out[b] = f;
        }
      }
    }
    __syncthreads();
  }
  const float* factors = fs.factors != nullptr ? fs.factors : sfac;
  const float4* p = reinterpret_cast<const float4*>(P) + static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x;
  const size_t stride = sample_stride / 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  constexpr int U = WIDE ? 4 : 8;
  int b = 0;
  if constexpr (WIDE) {
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    auto add = [&](float f, const float4& v) {
      const double c = static_cast<double>(f) * scale;
      sum[0] = fma(c, static_cast<double>(v.x), sum[0]); sum[1] = fma(c, static_cast<double>(v.y), sum[1]);
      sum[2] = fma(c, static_cast<double>(v.z), sum[2]); sum[3] = fma(c, static_cast<double>(v.w), sum[3]);
    };
    float4 v[U], w[U];
    auto fetch = [&](float4 (&to)[U]) {
#pragma unroll
      for (int k = 0; k < U; ++k) to[k] = __ldcs(p + k * stride);
      p += U * stride;
    };
    auto take = [&](const float4 (&from)[U]) {
#pragma unroll
      for (int k = 0; k < U; ++k) add(factors[b + k], from[k]);
      b += U;
    };
    // (the next samples' loads are under way while these are summed)
    const int groups = B / U;
    if (groups > 0) fetch(v);
    for (int g = 0; g < groups; g += 2) {
      if (g + 1 < groups) fetch(w);
      take(v);
      if (g + 1 >= groups) break;
      if (g + 2 < groups) fetch(v);
      take(w);
    }
    for (; b < B; ++b, p += stride) add(factors[b], __ldcs(p));
    acc = make_float4(static_cast<float>(sum[0]), static_cast<float>(sum[1]), static_cast<float>(sum[2]), static_cast<float>(sum[3]));
  } else {
    auto add = [&](float4& a, float c, const float4& v) {
      a.x = fmaf(c, v.x, a.x); a.y = fmaf(c, v.y, a.y); a.z = fmaf(c, v.z, a.z); a.w = fmaf(c, v.w, a.w);
    };
    for (; b + U <= B; b += U, p += U * stride) {
      float4 v[U], t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int k = 0; k < U; ++k) v[k] = __ldcs(p + k * stride);
#pragma unroll
      for (int k = 0; k < U; ++k) add(t, factors[b + k] * scale, v[k]);
      acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w;
    }
    for (; b < B; ++b, p += stride) add(acc, factors[b] * scale, __ldcs(p));
  }
  box[threadIdx.x >> 5][threadIdx.x & 31] = acc;
  __syncthreads();
  acc = box[threadIdx.x & 7][threadIdx.x >> 3];
  const int m = m0 + (threadIdx.x >> 3), n = n0 + (threadIdx.x & 7) * 4;
  if (m >= M || n >= N) return;
  const size_t idx = static_cast<size_t>(m) * N + n;
  float r[4] = {acc.x, acc.y, acc.z, acc.w};
  if (nk.std != 0.f) {
    if ((idx & 3) == 0) {
      float z[4];
      noise_group(nk, idx >> 2, z);
      r[0] += z[0]; r[1] += z[1]; r[2] += z[2]; r[3] += z[3];
    } else {     // a row pitch that is no multiple of four
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] += noise_at(nk, idx + j);
    }
  }
  if (vec_out) {     // N a multiple of four, `out` aligned to four elements
    if (out_dt == FDP_F32) {
      reinterpret_cast<float4*>(out)[idx >> 2] = make_float4(r[0], r[1], r[2], r[3]);
    } else if (out_dt == FDP_BF16) {
      const __nv_bfloat162 a = __floats2bfloat162_rn(r[0], r[1]), c = __floats2bfloat162_rn(r[2], r[3]);
      reinterpret_cast<uint2*>(out)[idx >> 2] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&c));
    } else {
      const __half2 a = __floats2half2_rn(r[0], r[1]), c = __floats2half2_rn(r[2], r[3]);
      reinterpret_cast<uint2*>(out)[idx >> 2] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&c));
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < N) store_as(out, out_dt, idx + j, r[j]);
  }
}

// ---- c_b pre-scale: Gs[r,:] = c[r / T] * G[r,:] (HBM-bound, 16-byte vectors) ------------------------
template <typename Tin>
__global__ void __launch_bounds__(256) prescale_kernel(const Tin* __restrict__ G, const float* __restrict__ factors,
                                                       Tin* __restrict__ Gs, size_t nvec, int vec_per_sample) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < nvec;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const float c = factors[i / vec_per_sample];
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(G) + i);
    const Tin* e = reinterpret_cast<const Tin*>(&raw);
    uint4 outv;
    Tin* o = reinterpret_cast<Tin*>(&outv);
#pragma unroll
    for (int v = 0; v < 8; ++v) o[v] = from_f32<Tin>(to_f32<Tin>(e[v]) * c);
    reinterpret_cast<uint4*>(Gs)[i] = outv;
  }
}

// ---- fp32 -> PLANES bf16 parts: dst[r, 0, c] = bf16(f x), dst[r, 1, c] = bf16(f x - hi), ..., with the column
// count rounded up to a multiple of 8 (zeros) and f a per-sample factor (1 when factors is null).  Both operands
// of a product in one launch: blocks below `first` work on job 0 ---------------------------------------------
struct SplitRun {
  const float* src; uint4* dst; const float* factors;
  unsigned nvec, vec_per_row;
  int n, T, vec;       // vec: n a multiple of 4, src 16-byte aligned
};
// MAXIMA: every block also leaves the largest magnitude that it has seen (as bits) in maxima[blockIdx.x], for simt_redo.
__device__ __forceinline__ unsigned magnitude(float f) { return __float_as_uint(f) & 0x7fffffffu; }
__device__ __forceinline__ unsigned block_max(unsigned v, unsigned* smem8) {      // 256 threads; valid in thread 0
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) smem8[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 1; i < 8; ++i) v = max(v, smem8[i]);
  return v;
}
template <int PLANES, bool MAXIMA>
__global__ void __launch_bounds__(256) split_kernel(const SplitRun j0, const SplitRun j1, unsigned first, int* zero_status, unsigned* maxima) {
  pdl_trigger();       // the product that follows sets itself up meanwhile
  if (zero_status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) { zero_status[0] = 0; zero_status[1] = 0; }   // (and split_stats_kernel's maximum)
  unsigned most = 0;
  const bool second = blockIdx.x >= first;
  const SplitRun& j = second ? j1 : j0;
  const unsigned block = second ? blockIdx.x - first : blockIdx.x, blocks = second ? gridDim.x - first : first;
  for (unsigned i = block * 256u + threadIdx.x; i < j.nvec; i += blocks * 256u) {
    const unsigned row = i / j.vec_per_row, cv = i - row * j.vec_per_row;
    const int c0 = static_cast<int>(cv) * 8;
    const float* p = j.src + static_cast<size_t>(row) * j.n + c0;
    float f[8];
    if (j.vec) {
      unpack16<float>(__ldg(reinterpret_cast<const uint4*>(p)), f);
      unpack16<float>(c0 + 4 < j.n ? __ldg(reinterpret_cast<const uint4*>(p) + 1) : make_uint4(0, 0, 0, 0), f + 4);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = c0 + e < j.n ? __ldg(p + e) : 0.f;
    }
    if (MAXIMA) {
#pragma unroll
      for (int e = 0; e < 8; ++e) most = max(most, magnitude(f[e]));
    }
    if (j.factors != nullptr) {
      const float c = __ldg(j.factors + row / j.T);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] *= c;
    }
    uint4* o = j.dst + static_cast<size_t>(row) * (PLANES * j.vec_per_row) + cv;
#pragma unroll
    for (int pl = 0; pl < PLANES; ++pl) {
      const uint4 h = pack16<__nv_bfloat16>(f);
      o[pl * j.vec_per_row] = h;
      float hf[8];
      unpack16<__nv_bfloat16>(h, hf);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] -= hf[e];
    }
  }
  if (MAXIMA) {
    __shared__ unsigned red[8];
    most = block_max(most, red);
    if (threadIdx.x == 0) maxima[blockIdx.x] = most;
  }
}

// ---- 16-bit operands whose rows are no multiple of 16 bytes: copies with padded rows (zeros), one or two in a launch --
// HBM-bound: one read, one write.  Eight elements a thread; a row's elements sit at any even address, so they are read
// as words where the columns are even in number and one by one otherwise (the lines come from L1).
__global__ void __launch_bounds__(256) pad_kernel(const SplitRun j0, const SplitRun j1, unsigned first, int* zero_status) {
  pdl_trigger();
  if (zero_status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *zero_status = 0;
  const bool second = blockIdx.x >= first;
  const SplitRun& j = second ? j1 : j0;
  const unsigned block = second ? blockIdx.x - first : blockIdx.x, blocks = second ? gridDim.x - first : first;
  const uint16_t* src = reinterpret_cast<const uint16_t*>(j.src);
  for (unsigned i = block * 256u + threadIdx.x; i < j.nvec; i += blocks * 256u) {
    const unsigned row = i / j.vec_per_row, cv = i - row * j.vec_per_row;
    const int c0 = static_cast<int>(cv) * 8;
    const uint16_t* p = src + static_cast<size_t>(row) * j.n + c0;
    uint32_t w[4];
    if (j.vec) {      // an even number of columns, 4-byte aligned
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = c0 + 2 * e < j.n ? __ldg(reinterpret_cast<const uint32_t*>(p) + e) : 0u;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t lo = c0 + 2 * e < j.n ? __ldg(p + 2 * e) : 0u, hi = c0 + 2 * e + 1 < j.n ? __ldg(p + 2 * e + 1) : 0u;
        w[e] = lo | (hi << 16);
      }
    }
    j.dst[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// ---- the split of G, with the bias gradient's statistics taken from the pass (grid and partials of gstats_kernel) ---
// In a whole backward G is split once for both products, and the column sums and sums of squares cost no read of
// their own: 8192 x 3072 fp32, G 33 + 33 + 23 us (two splits and the statistics) as separate passes, one pass here.
// MAXIMA: the largest magnitude goes to *maximum, which an earlier launch has cleared.
template <int PLANES, bool MAXIMA>
__global__ void __launch_bounds__(256, 4) split_stats_kernel(const float* __restrict__ G, uint2* __restrict__ dst,
                                                             float* __restrict__ colsum_part, float* __restrict__ sq_part,
                                                             int T, int n_out, int pitch, int rows_per_chunk,
                                                             int col_chunks, int row_chunks, unsigned* maximum) {
  pdl_trigger();
  unsigned most = 0;
  __shared__ float cs[8][32 * 4];
  __shared__ float red[32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int cc = blockIdx.x % col_chunks, rc = (blockIdx.x / col_chunks) % row_chunks;
  const int b = blockIdx.x / (col_chunks * row_chunks);
  const int c0 = (cc * 32 + x) * 4;
  const int r0 = rc * rows_per_chunk, r1 = min(T, r0 + rows_per_chunk);
  float acc[4] = {0.f, 0.f, 0.f, 0.f}, sq = 0.f;
  if (c0 < n_out) {
    const bool pad = c0 + 4 == n_out && pitch > n_out;
    auto take = [&](int r, const float4& v) {
      float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[e] += f[e]; sq = fmaf(f[e], f[e], sq);
        if (MAXIMA) most = max(most, magnitude(f[e]));
      }
      uint2* o = dst + ((static_cast<size_t>(b) * T + r) * PLANES * pitch + c0) / 4;
#pragma unroll
      for (int pl = 0; pl < PLANES; ++pl) {
        const __nv_bfloat162 h0 = __floats2bfloat162_rn(f[0], f[1]), h1 = __floats2bfloat162_rn(f[2], f[3]);
        o[pl * pitch / 4] = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
        if (pad) o[pl * pitch / 4 + 1] = make_uint2(0u, 0u);
        f[0] -= __low2float(h0); f[1] -= __high2float(h0); f[2] -= __low2float(h1); f[3] -= __high2float(h1);
      }
    };
    constexpr int U = 4;
    int r = r0 + y;
    for (; r + 8 * (U - 1) < r1; r += 8 * U) {
      float4 v[U];
#pragma unroll
      for (int k = 0; k < U; ++k) v[k] = __ldg(reinterpret_cast<const float4*>(G + (static_cast<size_t>(b) * T + r + 8 * k) * n_out + c0));
#pragma unroll
      for (int k = 0; k < U; ++k) take(r + 8 * k, v[k]);
    }
    for (; r < r1; r += 8) take(r, __ldg(reinterpret_cast<const float4*>(G + (static_cast<size_t>(b) * T + r) * n_out + c0)));
  }
#pragma unroll
  for (int v = 0; v < 4; ++v) cs[y][x * 4 + v] = acc[v];
  sq = block_sum(sq, red);  // contains the __syncthreads that publishes cs
  if (threadIdx.x == 0) sq_part[blockIdx.x] = sq;
  for (int c = threadIdx.x; c < 128; c += 256) {
    const int col = cc * 128 + c;
    if (col < n_out) {
      float t = 0.f;
#pragma unroll
      for (int yy = 0; yy < 8; ++yy) t += cs[yy][c];
      colsum_part[(static_cast<size_t>(b) * row_chunks + rc) * n_out + col] = t;
    }
  }
  if (MAXIMA) {
    __shared__ unsigned mred[8];
    most = block_max(most, mred);
    if (threadIdx.x == 0 && most > *static_cast<volatile unsigned*>(maximum)) atomicMax(maximum, most);
  }
}

// ---- host side ------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static std::mutex mu;
  static EncodeTiledFn fn = nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    else
      cudaGetLastError();
  }
  return fn;
}

// 2-D map over a row-major [rows, cols] matrix of 16-bit elements, 128-byte swizzle, zero fill
// (rows of `pitch` elements, 0: as many as there are columns)
bool make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_cols,
              uint32_t box_rows, int dt, uint64_t pitch = 0) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {(pitch != 0 ? pitch : cols) * 2};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(m, dt == FDP_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                        const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// [B * T, cols] as (column, row of the sample, sample), for K ranges that run over the rows: boxes of 64 x BK
bool make_rows_map(CUtensorMap* m, const void* base, int B, uint64_t T, uint64_t cols, int dt, uint64_t pitch = 0) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[3] = {cols, T, static_cast<cuuint64_t>(B)};
  if (pitch == 0) pitch = cols;
  const cuuint64_t strides[2] = {pitch * 2, pitch * 2 * T};
  const cuuint32_t box[3] = {64, BK, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(m, dt == FDP_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                        const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}
int pitch8(int n) { return (n + 7) & ~7; }     // columns of one part in a split copy
// three parts of [rows, cols] as (column, part, row), for products whose K range runs over the columns or over the rows
// of any number: what lies past the last of either reads as zeros
bool make_parts_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  const uint64_t pitch = pitch8(static_cast<int>(cols));
  const cuuint64_t dims[3] = {cols, 3, rows};
  const cuuint64_t strides[2] = {pitch * 2, 3 * pitch * 2};
  const cuuint32_t box[3] = {64, 1, box_rows};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Map of an output matrix [rows, cols] for the epilogue warps' boxes of 32 rows x 128 bytes.  The row pitch
// has to be a multiple of 16 bytes and the base 16-byte aligned.
bool make_out_map(CUtensorMap* m, void* base, uint64_t rows, uint64_t cols, int dt) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * dtype_size(dt)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / dtype_size(dt)), BOX_ROWS};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(m, dt == FDP_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : dt == FDP_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                                              : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                        2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

uint32_t make_idesc(int dt, bool a_mn, bool b_mn, int ctas = 1, int n = BN) {
  uint32_t d = 0;
  d |= 1u << 4;                                   // accumulator format: F32
  d |= (dt == FDP_BF16 ? 1u : 0u) << 7;           // A format
  d |= (dt == FDP_BF16 ? 1u : 0u) << 10;          // B format
  d |= (a_mn ? 1u : 0u) << 15;                    // A major: 1 = MN-major
  d |= (b_mn ? 1u : 0u) << 16;                    // B major
  d |= static_cast<uint32_t>(n >> 3) << 17;       // N
  d |= static_cast<uint32_t>((BM * ctas) >> 4) << 24;  // M (256 for a CTA pair)
  return d;
}

// SMs of the current device (cached per device).
int sm_count() {
  static std::mutex mu;
  static int cache[64];
  static bool have[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return 148; }
  std::lock_guard<std::mutex> lk(mu);
  if (!have[dev]) {
    int n = 148;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) { cudaGetLastError(); n = 148; }
    cache[dev] = n; have[dev] = true;
  }
  return cache[dev];
}
// SMs the next persistent GEMM grid may occupy: all of them minus the current reservation
// (fdp_set_sm_reserve; FDP_TC_RESERVE_SMS is its initial value).  A persistent CTA holds a whole SM's
// shared memory, so a collective kernel launched beside such a grid cannot start until SMs are free;
// a caller that overlaps a GEMM with a collective reserves a few SMs for the duration of that call.
std::atomic<int> g_sm_reserve{[] { const char* e = getenv("FDP_TC_RESERVE_SMS"); return e ? atoi(e) : 0; }()};
int launch_sms() {
  int n = sm_count();
  const int reserve = g_sm_reserve.load(std::memory_order_relaxed);
  if (n > MAX_SMS) n = MAX_SMS;   // the parking area is sized for MAX_SMS workers
  if (reserve > 0 && n - reserve >= 16) n -= reserve;
  return n & ~1;  // CTA pairs
}

template <bool A_MN, bool B_MN, int EPI, int CTAS = 1>
int launch(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& a2, const CUtensorMap& b2,
           const CUtensorMap& out, const TcArgs& args, cudaStream_t s) {
  static std::mutex mu;
  static bool done[64];
  constexpr int SMEM = smem_for(EPI);
  if (!smem_opt_in(done, mu, tc_gemm_kernel<A_MN, B_MN, EPI, CTAS>, SMEM)) return FDP_ERR_LAUNCH;
  TcArgs la = args;
  la.sticky = sticky_status_slot();
  const int total = la.batch * la.tiles_per_batch;
  if (la.cut != 2) la.cut = 1;
  if (la.split <= 1) { la.split = 1; if (la.cut == 1 && !la.park_whole) la.units_full = total; }
  int units = la.units_full + (total - la.units_full) * la.split * la.cut;
  const int workers = launch_sms() / CTAS;   // CTAs, or CTA pairs
  const int grid = CTAS * (units < workers ? units : workers);
  const bool dependent = la.dependent != 0 && pdl_enabled();
  if (CTAS == 1 && !dependent) {
    tc_gemm_kernel<A_MN, B_MN, EPI, CTAS><<<grid, threads_for(EPI), SMEM, s>>>(a, b, a2, b2, out, la);
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads_for(EPI));
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (CTAS == 2) {
      attr[na].id = cudaLaunchAttributeClusterDimension;
      attr[na].val.clusterDim.x = 2; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
      ++na;
    }
    if (dependent) {
      attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[na].val.programmaticStreamSerializationAllowed = 1;
      ++na;
    }
    cfg.attrs = attr; cfg.numAttrs = na;
    if (cudaLaunchKernelEx(&cfg, tc_gemm_kernel<A_MN, B_MN, EPI, CTAS>, a, b, a2, b2, out, la) != cudaSuccess) {
      cudaGetLastError();
      return FDP_ERR_LAUNCH;
    }
  }
  note_launch();
  return cudaPeekAtLastError() == cudaSuccess ? FDP_OK : (cudaGetLastError(), FDP_ERR_LAUNCH);
}

// CTA pairs (cta_group::2) for the store-epilogue GEMMs; FDP_TC_CTAS=1 / 2 forces single CTAs / pairs
int forced_ctas() {
  static const int v = [] { const char* e = getenv("FDP_TC_CTAS"); return (e && (e[0] == '1' || e[0] == '2')) ? e[0] - '0' : 0; }();
  return v;
}
int ctas_per_tile() { return forced_ctas() == 1 ? 1 : 2; }
// (Tried for the clipped-sum GEMM of small layers: single-CTA 128 x 256 tiles run whole, without K split,
// parked accumulators or fix-up, whenever the pair tiles do not fill one wave of CTA pairs.  At the four
// GPT-2-medium layer shapes that was 1-3 % slower than pairs with the K split, so pairs stay.)

// K-split of the tail wave: `rem` tiles left after the full waves (all of them when there are fewer
// tiles than workers) are cut into s parts of equal K-stage count, so that the last round keeps more
// SMs busy; cost in tile-times = ceil(rem*s/workers)/s plus the cost of parking and re-reading the
// accumulators.  At most 2 * workers parked parts (workers <= MAX_SMS / CTAS).
// That cost, in K stages of bf16 (0.40 us each when it was taken): 6 for the fix-up launch, 0.11 per part that it reads back
// (256 KB), 4 for each further round.  Measured, GEMM + fix-up: 48 pair tiles of 256 stages for 74 pairs 110 us
// unsplit, 117 in two parts, 91 in three; 16 tiles of 128 stages 54 / 37 / 30 / 26 us in one to four parts; 64 tiles
// of 128 stages 62 us unsplit, 72 in two parts.
int plan_tail_split(int total_tiles, int k_stages, int workers, int products, double whole = 1.0, double least_gain = 0.03,
                    int most_rounds = 2) {
  const int rem = total_tiles <= workers ? total_tiles : total_tiles % workers;
  // stages are counted by their work: with split fp32 operands one holds three or six products
  const int min_stages = products == 6 ? 2 : products == 3 ? 3 : 8;      // shortest part
  if (rem == 0 || k_stages < 4 * min_stages) return 1;
  // FDP_TC_SPLIT=n forces the number of parts (measurements), within the same limits
  static const int forced = [] { const char* e = getenv("FDP_TC_SPLIT"); return e ? atoi(e) : 0; }();
  if (forced >= 1) return (rem * forced > most_rounds * workers || k_stages / forced < min_stages) ? 1 : forced;
  int best_s = 1; double best = whole - least_gain + 0.03;     // `whole`: tile-times of the round without a split
  for (int sp = 2; sp <= 16; ++sp) {
    if (rem * sp > most_rounds * workers || k_stages / sp < min_stages) break;
    const int rounds = (rem * sp + workers - 1) / workers;
    const double cost = static_cast<double>(rounds) / sp +
                        (6.0 + 0.11 * rem * sp + 4.0 * (rounds - 1)) / (static_cast<double>(k_stages) * products);
    if (cost < best - 0.03) { best = cost; best_s = sp; }
  }
  return best_s;
}
// The last round of the forward and input-gradient products.  Tiles that fill less than half of it (all of them where
// there are fewer than half the workers) are cut in two along N, so that the round takes less: 6000 rows 4096 -> 1024 fp16,
// 96 tiles for 74 pairs, 46.2 -> 41.6 us; 192 rows 1216 -> 384 bf16, 2 tiles, 13.0 -> 8.8; 512 rows 768 -> 768 fp32,
// 6 tiles, 19.6 -> 14.9.  Or, with a place to park the parts, the tiles are cut along K where that takes less still:
// a narrow stage takes 0.7 of a whole one (its copies are 0.75), another launch is worth ten stages, and
// parts of more than one round gain nothing (3152 rows 3072 -> 768 fp32, 39 tiles in three parts: 61.2 / 60.3 us).  972 rows 3480 -> 688
// bf16, 12 tiles of 55 stages, 22.3 -> 15.5 us; 300 rows 8192 -> 264 30.2 -> 21.2; fp32 in six products 2816 rows 3888 -> 64
// 86 -> 48, 128 rows 8190 -> 70 119 -> 34.
int plan_gemm_split(int total, int k_stages, int workers, int products) {
  const int rem = total <= workers ? total : total % workers;
  return plan_tail_split(total, k_stages, workers, products, 2 * rem <= workers ? 0.7 : 1.0, 10.0 / (static_cast<double>(k_stages) * products), 1);
}
// parking space of a product; a constant SM count, like every plan that a workspace query shares with the launch
size_t gemm_park_bytes(int rows, int K, int N, int products) {
  const int ctas = ctas_per_tile(), workers = MAX_SMS / ctas;
  const int total = ceil_div(rows, BM * ctas) * ceil_div(N, BN), rem = total <= workers ? total : total % workers;
  const int split = plan_gemm_split(total, ceil_div(K, BK), workers, products);
  return split <= 1 ? 0 : static_cast<size_t>(rem) * split * ctas * BM * BN * sizeof(float);
}
// `mp`: map of the parking space, where it is used
bool plan_last_round(TcArgs& a, int ctas, uint32_t idesc_half, int K, int products, const GemmPark& park, CUtensorMap* mp) {
  const int total = a.tiles_per_batch;
  const size_t bytes = gemm_park_bytes(a.M, K, a.N, products);
  if (bytes > 0 && park.ws != nullptr && park.bytes >= bytes) {
    const int workers = MAX_SMS / ctas, rem = total <= workers ? total : total % workers;
    a.split = plan_gemm_split(total, a.k_stages, workers, products);
    a.units_full = total - rem;
    a.split_ws = park.ws;
    return make_out_map(mp, park.ws, bytes / (BN * sizeof(float)), BN, FDP_F32);
  }
  const int workers = launch_sms() / ctas, rem = total <= workers ? total : total % workers;
  if (ctas != 2 || rem == 0 || 2 * rem > workers) return true;
  a.cut = 2; a.units_full = total - rem; a.idesc_half = idesc_half;
  return true;
}
// the parts of a K split into their tiles
int gemm_fixup(int st, const TcArgs& a, int ctas, cudaStream_t s) {
  if (st != FDP_OK || a.split <= 1) return st;
  launch_dependent(splitk_fixup_kernel, dim3(BM * ctas * BN / (256 * 4), a.tiles_per_batch - a.units_full), dim3(256), 0, s, a.split_ws,
                   a.units_full, a.split, BM * ctas, a.M, a.N, a.tiles_m, a.tiles_n, a.n_fastest, a.m_group, a.out, a.out_dt, a.ld_out,
                   1.0f, a.nk, a.bias, a.bias_dt);
  note_launch();
  return cudaPeekAtLastError() == cudaSuccess ? FDP_OK : (cudaGetLastError(), FDP_ERR_LAUNCH);
}
// parked accumulators: up to 2 * MAX_SMS parts of 128 x 256 fp32 (a CTA pair parks two per part)
size_t split_ws_bytes() { return static_cast<size_t>(2) * MAX_SMS * BM * BN * sizeof(float); }
size_t align256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

int gram_tiles(int T) { return gram_units(ceil_div(T, BM)); }   // work units (128 x 256 tiles) per sample

// A warp waits on a barrier nobody arrives on, so the wait runs out after `limit` cycles and takes the
// reporting path of every bounded wait of the library: abort flag, status word, host-visible slot.
__global__ void __launch_bounds__(32) wait_selftest_kernel(int* status, int* sticky, long long limit) {
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) { mbar_init(smem_u32(&bar), 1); abort_flag = 0; mbar_fence_init(); }
  __syncwarp();
  const WaitCtx w{&abort_flag, status, sticky, limit};
  mbar_wait_warp(smem_u32(&bar), 0, w, 9);
}

}  // namespace

int sm_reserve_exchange(int n) { return g_sm_reserve.exchange(n < 0 ? 0 : n); }

int tc_wait_selftest(int* status, long long limit_cycles, cudaStream_t s) {
  if (limit_cycles < 1) limit_cycles = 1;
  if (limit_cycles > WAIT_LIMIT_CYCLES) limit_cycles = WAIT_LIMIT_CYCLES;
  wait_selftest_kernel<<<1, 32, 0, s>>>(status, sticky_status_slot(), limit_cycles);
  note_launch();
  return cudaPeekAtLastError() == cudaSuccess ? FDP_OK : (cudaGetLastError(), FDP_ERR_LAUNCH);
}

// K stages per accumulator hand-off for fp32 inputs (a stage = 12 MMA steps of K = 16, three products of
// four): FDP_TC_CHAIN_STAGES, default 2.  B=8, T=1024, 4096x4096 against float64, 1 / 2 / 3 / 4 / 8 stages:
// norms off by 2.0e-7 / 3.8e-7 / 5.2e-7 / 7.3e-7 / 1.4e-6 (the truncation of the accumulators grows with the
// chain); B=8, T=1024, 1024->3072, all kernels of a forward and backward: 832 / 636 / 616 / 592 / 588 us.
// Six products (24 steps a stage, of which only the four of hi*hi meet a large accumulator): one stage.
static int chain_stages(int seg_stages, int planes) {
  if (planes == 3) return 1;
  static const int cap = [] {
    const char* e = getenv("FDP_TC_CHAIN_STAGES");
    const int v = e ? atoi(e) : 2;
    return v < 1 ? 1 : v;
  }();
  return cap < seg_stages ? cap : seg_stages;
}

// ... and for 16-bit products that are kept: 8 stages, 32 truncated steps.  16 x 1024 rows, 1024 -> 3072, weight gradient with one
// accumulator a sample 122 us, in chains of 8 / 4 / 2 stages 125 / 131 / 138; 1 x 4096, 1024 -> 1024, clipping off, error of dW
// 4.4e-6 with one, 4.8e-7 with 8 stages, and 1.0e-6 when it was contracted twice and cut along K.
constexpr int KEPT_CHAIN = 8;
static int kept_chain(int seg_stages, bool pad) {
  const int n = pad ? 1 : KEPT_CHAIN;
  return n < seg_stages ? n : seg_stages;
}

// fp32 shapes of FDP_FP32_TENSOR's three products: whole 64-column and 64-row K stages, at least 128 of everything
static bool three_products_ok(int T, int n_in, int n_out) {
  return n_in % BK == 0 && n_out % BK == 0 && n_in >= 128 && n_out >= 128 && T % BK == 0 && T >= 2 * BK;
}

// ... and of FDP_FP32_WIDE's six
static bool wide_ok(int B, int T, int n_in, int n_out, int norm_algo) {
  if (n_in < 64 || n_out < 64) return false;
  // T >= 64: the FMA kernels lose at every size, one sample of 64 rows included (whole call, 64 -> 64: 24.7 us, six
  // products 15.8; 1024 -> 1000: 219 / 18.5; 8192 -> 8200: 1945 / 152).  Shorter sequences have no norm pass on the tensor
  // cores to gain from, and below 128 rows in all the FMA kernels' K loop is shorter than the extra launches: 64 samples
  // of one row, 256 -> 256, 43 us a call against 52; 210 rows, 1024 -> 4096, 122 against 77.
  return T >= SHORT_SEQ || (norm_algo != FDP_NORM_DIRECT && static_cast<long long>(B) * T >= 128);
}

// tiles of a sample's product, in the orientation that has more (the workspace query does not know the layout)
static int most_product_tiles(int n_in, int n_out) {
  const int ctas = ctas_per_tile();
  const int a = ceil_div(n_out, BM * ctas) * ceil_div(n_in, BN), b = ceil_div(n_in, BM * ctas) * ceil_div(n_out, BN);
  return a > b ? a : b;
}
// norm partials per sample of a product pass that keeps nothing: always in the orientation [out, in] (tc_norms)
static int product_partials(int n_in, int n_out) {
  const int ctas = ctas_per_tile();
  return ceil_div(n_out, BM * ctas) * ceil_div(n_in, BN) * ctas * epi_warps_for(EPI_STORE_SCALED);
}
// K stages of a sample over which six products that are kept are summed at once (two additions a stage): half of what a part
// of the contraction would sum that they take the place of (one a stage).  Error of dW against float64, contracted twice / summed
// at once / so: 9 x 2432 rows, 360 -> 835 1.5e-7 / 1.7e-7 / 1.3e-7; 8 x 3264, 128 -> 136 1.4e-7 / 1.9e-7 / 1.3e-7; 2 x 936,
// 448 -> 1368 9.2e-8 / 1.25e-7 / 9.9e-8.  A visit to the kept tile takes 2 to 3 us: never for less than four stages (8 x 3264 102 us, now
// 109; 5 x 704, 1344 -> 64 35 / 41; contracted twice 173 and 53).
static int part_stages(int B, int stages, int n_in, int n_out, int products);
static int kept_flush(int B, int stages, int n_in, int n_out) {
  const int n = part_stages(B, stages, n_in, n_out, 6) / 2;
  return n < 4 ? 4 : n;
}
static size_t keep_bytes(int B, int n_in, int n_out) {
  return static_cast<size_t>(B) * most_product_tiles(n_in, n_out) * ctas_per_tile() * BM * BN * sizeof(float);
}
// ---- estimates in us by which weight-gradient plans are chosen -----------------------------------------------------
// Fitted to 36 shapes, B 1 to 64, T 64 to 4096, widths 64 to 11008, every side timed, when a CTA pair took 0.30 us a K stage and
// an accumulator's return held it up (0.19 now): as times they are too high by up to a half, on all sides.  What they are for
// was timed again with the present kernels: of 315 shapes from T = 64 on the choice between kept and contracted twice is more
// than 5 % off at 7 (at worst 3 x 681 rows 1712 -> 5304 fp16, 77 us kept, 68 twice), of 419 shorter ones that between three plans
// more than 8 % off at 9 (at worst 1 x 3, 128 -> 192 fp32, blocks 18 us, kept 12).
// The SM count is a constant: the workspace query and the launch must pick the same plan.
namespace {
constexpr int PLAN_PAIRS = MAX_SMS / 2;
double rounds(long long units, int on) { return static_cast<double>((units + on - 1) / on); }
// every sample's product once, kept, and their weighted sum
double keep_us(int B, int T, int n_in, int n_out, int planes) {
  constexpr double STAGE[3] = {0.38, 1.22, 2.9}, FIXED[3] = {1.8, 2.2, 2.2}, LEAST[3] = {3.5, 5.0, 5.0};
  const double r = ceil_div(T, BK) * STAGE[planes - 1] + FIXED[planes - 1], least = LEAST[planes - 1];
  // (a product of few boxes keeps few SMs at the sum, sample after sample: 590 x 1 rows, 195 -> 192 bf16 105 us, blocks 86, twice 59)
  const double hbm = 4.0 * n_in * n_out * (B + 1.0) / 6.4e6, serial = 0.11 * B - 7.0;
  return 9.5 + rounds(static_cast<long long>(B) * most_product_tiles(n_in, n_out), PLAN_PAIRS) * (r > least ? r : least) +
         (hbm > serial ? hbm : serial);
}
// a norm pass over product tiles or Gram blocks
double norm_us(int B, int T, int n_in, int n_out, int planes, int algo) {
  const int stages = ceil_div(T, BK);
  if (planes > 1) {
    constexpr double STAGE[3] = {0.0, 1.05, 2.45}, FIXED[3] = {0.0, 0.5, 1.5};
    return 6.0 + rounds(static_cast<long long>(B) * most_product_tiles(n_in, n_out), PLAN_PAIRS) * (stages * STAGE[planes - 1] + FIXED[planes - 1]);
  }
  if (algo == FDP_NORM_DIRECT)
    return 4.0 + rounds(static_cast<long long>(B) * ceil_div(n_out, BM) * ceil_div(n_in, BN), MAX_SMS) * (stages * 0.42 + 1.0);
  return 4.0 + rounds(static_cast<long long>(B) * gram_tiles(T), MAX_SMS) * ((ceil_div(n_in, BK) + ceil_div(n_out, BK)) * 0.40 + 1.0);
}
// the clipped sum as one contraction, factors per sample in the epilogue (`scaled`) or in a copy of G
double sum_us(int B, int T, int n_in, int n_out, int planes, bool scaled) {
  constexpr double STAGE[3] = {0.40, 1.2, 2.2};
  const int tiles = most_product_tiles(n_in, n_out);
  const int k = scaled ? B * ceil_div(T, BK) : static_cast<int>((static_cast<long long>(B) * T + BK - 1) / BK);
  const int split = plan_tail_split(tiles, k, PLAN_PAIRS, planes == 3 ? 6 : planes == 2 ? 3 : 1);
  const int rem = tiles <= PLAN_PAIRS ? tiles : tiles % PLAN_PAIRS;
  const double waves = (tiles - rem) / PLAN_PAIRS + rounds(static_cast<long long>(rem) * split, PLAN_PAIRS) / split;
  double us = 6.0 + waves * (k * STAGE[planes - 1] + (scaled && planes == 1 ? 0.5 * B : 0.0));
  if (split > 1) us += 4.0 + 0.04 * rem * split;
  if (!scaled) us += 4.5 + 4.0 * B * T * n_out / 5e6;
  return us;
}
// norms of short samples by the T x T blocks of simt_norm_gram_small, one block a sample: 4 x 10 rows, 7400 + 72 columns
// 129 us, 46 x 27, 6272 + 176 309, 2 x 40, 7248 + 256 391, 2 x 3, 6848 + 123 105
double small_norm_us(int B, int T, int cols) {
  if (T == 1) return 4.0;
  const double waves = B > 400 ? B / 400.0 : 1.0;
  return 3.0 + waves * cols * (0.015 + T * T / 31000.0);
}
// the clipped sum on FMA kernels: 42 rows 1472 -> 2496 34 us, 40 rows 7400 -> 72 20, 17 rows 6904 -> 2308 64
double fma_sum_us(long long rows, int n_in, int n_out) {
  const double waves = static_cast<double>(ceil_div(n_in, 64)) * ceil_div(n_out, 64) / MAX_SMS;
  return 5.0 + rows * 0.14 * (waves > 1.0 ? waves : 1.0);
}
}  // namespace

// K stages in a part of the clipped sum's contraction
static int part_stages(int B, int stages, int n_in, int n_out, int products) {
  return B * stages / plan_tail_split(most_product_tiles(n_in, n_out), B * stages, PLAN_PAIRS, products);
}
// Whether keeping the per-sample products beats the plan `p` that contracts twice.  They part where B n_in n_out fp32
// elements written and read cost what a norm pass costs: 8 x 1024 rows 1024 -> 3072 bf16 66 us kept, 76 contracted twice,
// 1024 -> 1024 27 / 38; fp32 (three products) 8 x 1024, 1024 -> 3072 170 / 252; 12 x 500, 1024 -> 4096 fp16 (67 us) and 16 x 512,
// 4096 -> 4096 bf16 (238) are contracted twice.
static bool keep_wins(int B, int T, int n_in, int n_out, const TcPlan& p) {
  if (keep_bytes(B, n_in, n_out) > KEEP_LIMIT) return false;
  // 16-bit samples of few rows leave faster than they can be written (64 x 128 rows, 1024 -> 1024: 101 us kept, 47; 48 x 64,
  // 768 -> 3072: 160 / 53); only calls of a few launches gain there (5 x 92, 512 -> 512: 12.6 / 18.6), which the host bounds.
  if (p.planes == 1 && !p.pad && T < 256) return false;
  // No precision is given up for it.  Contracted twice, a tile that is cut along K holds its sums in as many accumulators;
  // kept, a sample's sum is one: its chain of truncating additions (kept_chain) may not be longer than what a part sums.  (Six
  // products: kept_flush.)  And the Gram form of the norms has chains of n_in and n_out (bf16 norms from float64, Gram / one
  // accumulator a sample: 2 x 1024 rows, 256 -> 256 3.9e-7 / 8.5e-7; 1 x 2560, 3624 -> 1288 6.2e-6 / 2.3e-6).
  const int stages = ceil_div(T, BK);
  if (p.planes == 1 && p.scaled_epilogue && kept_chain(stages, p.pad) > part_stages(B, stages, n_in, n_out, 1)) return false;
  if (p.algo == FDP_NORM_GRAM && BK * kept_chain(stages, p.pad) > n_in + n_out) return false;
  // (fp32 calls hold the parts of both operands already: a tenth has to be gained for more)
  return keep_us(B, T, n_in, n_out, p.planes) < (p.planes > 1 ? 0.9 : 0.97) * (norm_us(B, T, n_in, n_out, p.planes, p.algo) +
                                                                             sum_us(B, T, n_in, n_out, p.planes, p.scaled_epilogue));
}

// Turns `p` into a plan that keeps the products.  With split fp32 operands never in less than the parking area: a call that
// is short of memory gives way where it did before.
static void plan_keep(TcPlan& p, int B, int n_in, int n_out) {
  p.ok = true; p.keep = true; p.short_seq = false; p.scaled_epilogue = false; p.algo = FDP_NORM_DIRECT;
  p.nparts = most_product_tiles(n_in, n_out) * ctas_per_tile() * epi_warps_for(EPI_CHAIN_SUMSQ);
  p.split_bytes = keep_bytes(B, n_in, n_out);
  if (p.planes > 1 && p.split_bytes < split_ws_bytes()) p.split_bytes = split_ws_bytes();
  p.ws_bytes = p.split_bytes + p.split_g_bytes + p.split_x_bytes + p.pad_g_bytes + p.pad_x_bytes;
}

// Short samples (T < SHORT_SEQ): `p` has norms by T x T blocks and a pre-scaled contraction, or nothing (p.ok unset: the FMA
// kernels).  Both are slow for few samples of wide layers, one block a sample: instead the product form of longer samples,
// their one K stage filled up with zeros, kept or contracted twice, where that is expected to take less.  3 x 44 rows,
// 1024 -> 3072 bf16: 266 us, now 14; 40 x 20, 1000 -> 1000 fp32 85 / 58; 64 x 16, 1024 -> 1024 bf16 47 / 41; 1000 x 30,
// 768 -> 768 stays (282).
static void plan_short(TcPlan& p, int B, int T, int n_in, int n_out) {
  const double before = small_norm_us(B, T, n_in + n_out) + 2.0 +
                        (p.ok ? sum_us(B, T, n_in, n_out, p.planes, false) : fma_sum_us(static_cast<long long>(B) * T, n_in, n_out));
  const double kept = keep_bytes(B, n_in, n_out) <= KEEP_LIMIT ? keep_us(B, T, n_in, n_out, p.planes) : 1e30;
  const double twice = norm_us(B, T, n_in, n_out, p.planes, FDP_NORM_DIRECT) + sum_us(B, T, n_in, n_out, p.planes, true);
  if ((kept < twice ? kept : twice) > 0.9 * before) return;
  if (kept < twice) { plan_keep(p, B, n_in, n_out); return; }
  p.ok = true; p.short_seq = false; p.scaled_epilogue = true; p.algo = FDP_NORM_DIRECT;
  p.nparts = p.planes > 1 || p.pad ? product_partials(n_in, n_out)
                                   : 4 * ceil_div(n_out, BM) * ceil_div(n_in, BN);
  p.split_bytes = split_ws_bytes();
  p.ws_bytes = p.split_bytes + p.split_g_bytes + p.split_x_bytes + p.pad_g_bytes + p.pad_x_bytes;
}

// (16-bit inputs without FDP_PAD_16BIT: row pitches that are multiples of 16 bytes, and matrices large enough that the
// 128 x 256 tile is not mostly padding)
TcPlan tc_plan(int B, int T, int n_in, int n_out, int dt, int norm_algo) {
  TcPlan p; p.ok = false; p.algo = FDP_NORM_DIRECT; p.ws_bytes = 0; p.nparts = 0; p.scaled_epilogue = false;
  p.short_seq = false; p.any_align = false; p.keep = false; p.split_bytes = 0;
  p.planes = 1; p.split_g_bytes = p.split_x_bytes = 0;
  p.pad = false; p.pad_g_bytes = p.pad_x_bytes = 0;
  const bool fp32_tensor = (norm_algo & FDP_FP32_TENSOR) != 0, fp32_wide = (norm_algo & FDP_FP32_WIDE) != 0;
  const bool may_pad = (norm_algo & FDP_PAD_16BIT) != 0;
  const bool may_keep = (norm_algo & (FDP_KEEP_PRODUCTS | FDP_NORM_MASK)) == (FDP_KEEP_PRODUCTS | FDP_NORM_AUTO);
  norm_algo &= FDP_NORM_MASK;
  if (dt == FDP_F32) {
    // fp32 on the tensor cores, when the caller asks for it.  FDP_FP32_TENSOR: three bf16 products (hi*hi +
    // hi*lo + lo*hi).  FDP_FP32_WIDE: six products over three parts for the shapes the former does not take --
    // any width (the split copies have padded rows), any T -- because those ran on FMA kernels and their
    // results are to be no further from float64 than FMA ones.  The tensor cores add into their fp32
    // accumulators by truncation, a one-sided error of about 2^-24 per K=16 step, so no accumulator runs for
    // more than a few K stages: it is handed to the epilogue warps, which add it to registers with
    // round-to-nearest (chain_stages).  The clip factors are applied there per sample (or, for short
    // sequences, in fp32 before the split: a pre-scaled bf16 copy would round c_b * G).
    const bool wide = fp32_wide && wide_ok(B, T, n_in, n_out, norm_algo);
    if (fp32_tensor && three_products_ok(T, n_in, n_out)) p.planes = 2;
    else if (wide || (fp32_wide && may_keep && T < SHORT_SEQ && n_in >= 64 && n_out >= 64)) p.planes = 3;
    else return p;
    p.any_align = p.planes == 3;
    p.split_g_bytes = align256(static_cast<size_t>(B) * T * pitch8(n_out) * 2 * p.planes);
    p.split_x_bytes = align256(static_cast<size_t>(B) * T * pitch8(n_in) * 2 * p.planes);
    p.split_bytes = split_ws_bytes();
    p.ws_bytes = p.split_bytes + p.split_g_bytes + p.split_x_bytes;
    if (T < SHORT_SEQ) {
      p.algo = FDP_NORM_GRAM; p.short_seq = true; p.nparts = 1;
      p.ok = wide;
      if (may_keep) plan_short(p, B, T, n_in, n_out);
      return p;
    }
    // always the product form, accumulated in short chains (tc_norms); the Gram form needs both T x T tiles
    // complete in TMEM before its epilogue can multiply them, i.e. one chain of 3 * (in + out) / 16
    // truncating additions.  The chained norm pass: tiles of the clipped-sum GEMM, eight epilogue warps per CTA
    p.ok = true; p.algo = FDP_NORM_DIRECT; p.scaled_epilogue = true;
    p.nparts = product_partials(n_in, n_out);
    if (may_keep && keep_wins(B, T, n_in, n_out, p)) plan_keep(p, B, n_in, n_out);
    return p;
  }
  if (dt != FDP_BF16 && dt != FDP_F16) return p;
  if (n_in % 8 != 0 || n_out % 8 != 0 || n_in < 128 || n_out < 128) {
    // Any width from 64 on with FDP_PAD_16BIT: operands whose rows (or pointers) are no multiple of 16 bytes are copied.
    // The FMA kernels that these shapes ran on apply the factors in fp32 and add in short chains, so G is never pre-scaled
    // here and no accumulator runs for more than a stage.  Whole weight gradients, error of dW and of the norms against
    // float64: 30 x 768 rows 5952 -> 64 bf16 5124 us, 2.7e-6, 7e-8 before, now 85 us, 1.3e-7, 1.0e-7; 16 x 1024, 1023 -> 3071
    // 10168 / 220 us; 64 x 256, 65 -> 66 2063 / 28; 3 x 300, 129 -> 1001 fp16 144 / 15; 2 x 64, 64 -> 64 30 / 9.
    if (!may_pad || n_in < 64 || n_out < 64) return p;
    p.pad = true; p.any_align = true;
    p.pad_g_bytes = align256(static_cast<size_t>(B) * T * pitch8(n_out) * 2);
    p.pad_x_bytes = align256(static_cast<size_t>(B) * T * pitch8(n_in) * 2);
  }
  if (T < SHORT_SEQ) {
    // short sequences: the norms come from the small Gram kernel (one partial per sample); the
    // clipped sum is still one GEMM with K = B*T over the pre-scaled copy of G, if K is worth a tile
    if (norm_algo == FDP_NORM_DIRECT) return p;
    p.algo = FDP_NORM_GRAM; p.short_seq = true; p.nparts = 1;
    p.ok = !p.pad && static_cast<long long>(B) * T >= 4 * BK;
    p.split_bytes = split_ws_bytes();
    p.ws_bytes = p.split_bytes + align256(static_cast<size_t>(B) * T * n_out * 2);
    if (may_keep) plan_short(p, B, T, n_in, n_out);
    return p;
  }
  // Cost of the two norm algorithms in K stages on the critical path: both kernels deal equal work
  // units (128x256 tiles) round-robin to one CTA per SM, so a pass takes
  // ceil(units / SMs) * (stages per unit + a fixed cost per unit of about four stages).  The SM
  // count is a constant here: the workspace query and the launch must pick the same algorithm.
  constexpr long long PLAN_SMS = 148, UNIT_FIXED_STAGES = 4;
  const long long units_d = static_cast<long long>(B) * ceil_div(n_out, BM) * ceil_div(n_in, BN);
  const long long units_g = static_cast<long long>(B) * gram_tiles(T);
  const double direct = static_cast<double>((units_d + PLAN_SMS - 1) / PLAN_SMS) * (ceil_div(T, BK) + UNIT_FIXED_STAGES);
  const double gram = static_cast<double>((units_g + PLAN_SMS - 1) / PLAN_SMS) *
                      (ceil_div(n_in, BK) + ceil_div(n_out, BK) + UNIT_FIXED_STAGES);
  int algo = norm_algo;
  if (algo == FDP_NORM_AUTO) algo = direct <= gram ? FDP_NORM_DIRECT : FDP_NORM_GRAM;
  if (p.pad) algo = FDP_NORM_DIRECT;      // in chains of one stage, over the tiles of the clipped sum
  p.ok = true;
  p.algo = algo;
  // clip factors applied in the GEMM epilogue (no scaled copy of G) when a sample's main loop is long
  // enough to hide the per-sample drain and its last K stage is not mostly padding: the padded rows cost
  // pad * n_in * n_out multiply-adds a sample, the pre-scale pass reads and writes T * n_out elements, about
  // 400 multiply-adds' time each.  FDP_WGRAD_PRESCALE=1 forces the pre-scale pass (for A/B measurements)
  static const bool force_prescale = [] { const char* e = getenv("FDP_WGRAD_PRESCALE"); return e && e[0] == '1'; }();
  const long long pad = static_cast<long long>(ceil_div(T, BK)) * BK - T;
  p.scaled_epilogue = p.pad || (!force_prescale && T >= 256 && pad * n_in <= 400ll * T);
  // one partial per work unit and epilogue warp
  p.nparts = p.pad ? product_partials(n_in, n_out)
                   : 4 * ((algo == FDP_NORM_DIRECT) ? ceil_div(n_out, BM) * ceil_div(n_in, BN) : gram_tiles(T));
  // the parked accumulators of the split-K tail, then (pre-scale path only) the c_b-scaled copy of G
  p.split_bytes = split_ws_bytes();
  p.ws_bytes = p.split_bytes + (p.scaled_epilogue ? 0 : align256(static_cast<size_t>(B) * T * n_out * 2)) + p.pad_g_bytes + p.pad_x_bytes;
  if (may_keep && keep_wins(B, T, n_in, n_out, p)) plan_keep(p, B, n_in, n_out);
  return p;
}

int tc_split(const SplitJob* jobs, int njobs, int planes, int* zero_status, cudaStream_t s, unsigned* maxima, Maxima* of_job) {
  SplitRun r[2] = {};
  unsigned blocks[2] = {0, 0};
  // 32-bit index arithmetic within a launch: an operand past that is cut along its rows
  size_t done[2] = {0, 0};
  for (;;) {
    for (int k = 0; k < 2; ++k) {
      blocks[k] = 0;
      if (k >= njobs || done[k] >= jobs[k].rows) continue;
      const SplitJob& j = jobs[k];
      const unsigned vpr = pitch8(j.n) / 8;
      const size_t most = (1u << 31) / vpr, left = j.rows - done[k], nr = left < most ? left : most;
      if (nr < j.rows && j.factors != nullptr) return FDP_ERR_SHAPE;   // (factors come with short sequences only)
      // (planes 0: a 16-bit operand is copied as it is)
      r[k].src = reinterpret_cast<const float*>(static_cast<const char*>(j.src) + done[k] * j.n * (planes > 0 ? 4 : 2));
      r[k].dst = static_cast<uint4*>(j.dst) + done[k] * vpr * (planes > 0 ? planes : 1);
      r[k].factors = j.factors; r[k].T = j.T; r[k].n = j.n; r[k].vec_per_row = vpr;
      r[k].nvec = static_cast<unsigned>(nr * vpr);
      r[k].vec = planes > 0 ? j.n % 4 == 0 && aligned16(r[k].src) : j.n % 2 == 0 && reinterpret_cast<uintptr_t>(r[k].src) % 4 == 0;
      blocks[k] = (r[k].nvec + 255) / 256;
      done[k] += nr;
    }
    if (blocks[0] + blocks[1] == 0) break;
    // 16 blocks an SM in all, shared in proportion to the work
    const unsigned cap = static_cast<unsigned>(sm_count() < MAX_SMS ? sm_count() : MAX_SMS) * 16;
    const unsigned long long all = static_cast<unsigned long long>(blocks[0]) + blocks[1];
    if (all > cap) {
      for (int k = 0; k < 2; ++k)
        if (blocks[k] > 0) blocks[k] = static_cast<unsigned>(blocks[k] * static_cast<unsigned long long>(cap) / all) + 1;
    }
    if (planes == 0) pad_kernel<<<blocks[0] + blocks[1], 256, 0, s>>>(r[0], r[1], blocks[0], zero_status);
    else if (planes == 2) split_kernel<2, false><<<blocks[0] + blocks[1], 256, 0, s>>>(r[0], r[1], blocks[0], zero_status, nullptr);
    else if (maxima == nullptr) split_kernel<3, false><<<blocks[0] + blocks[1], 256, 0, s>>>(r[0], r[1], blocks[0], zero_status, nullptr);
    else split_kernel<3, true><<<blocks[0] + blocks[1], 256, 0, s>>>(r[0], r[1], blocks[0], zero_status, maxima);
    if (maxima != nullptr)       // (operands of one launch: tc_gemm6_ok)
      for (int k = 0; k < njobs; ++k) of_job[k] = Maxima{maxima + (k == 1 ? blocks[0] : 0), static_cast<int>(blocks[k])};
    note_launch();
  }
  return cudaPeekAtLastError() == cudaSuccess ? FDP_OK : (cudaGetLastError(), FDP_ERR_LAUNCH);
}

bool tc_split_stats_ok(const void* G, int n_out) { return n_out % 4 == 0 && aligned16(G); }
int tc_split_stats(const void* G, void* dst, float* colsum_part, float* sq_part, int B, int T, int n_out, int planes,
                   const GstatsPlan& pl, cudaStream_t s, unsigned* maximum) {
  const unsigned grid = static_cast<unsigned>(static_cast<size_t>(B) * pl.row_chunks * pl.col_chunks);
  auto kernel = planes == 2 ? split_stats_kernel<2, false> : maximum == nullptr ? split_stats_kernel<3, false> : split_stats_kernel<3, true>;
  kernel<<<grid, 256, 0, s>>>(static_cast<const float*>(G), static_cast<uint2*>(dst), colsum_part, sq_part, T, n_out, pitch8(n_out),
                              pl.rows_per_chunk, pl.col_chunks, pl.row_chunks, maximum);
  note_launch();
  return cudaPeekAtLastError() == cudaSuccess ? FDP_OK : (cudaGetLastError(), FDP_ERR_LAUNCH);
}

int tc_norms(const void* G, const void* X, float* partials, int* dev_status, int B, int T, int n_in,
             int n_out, int dt, const TcPlan& pl, cudaStream_t s, float* keep, int layout, int pitch_g, int pitch_x) {
  const uint64_t rows = static_cast<uint64_t>(B) * T;
  CUtensorMap a, b, a2, b2;
  TcArgs args{};
  args.batch = B; args.batch_rows = T; args.partials = partials; args.status = dev_status; args.T = T;
  args.zero_status = 1;      // the norm pass is the first launch of a weight-gradient call
  if (pl.planes > 1 || pl.pad || keep != nullptr) {
    // fp32 inputs, 16-bit ones that come as padded copies, and products that are kept: the per-sample products G_b^T X_b themselves, on the tiles and CTA pairs of the
    // clipped-sum GEMM, handed to the epilogue every few K stages and summed there in registers; a
    // unit is (sample, tile) and ends with the sum of its squares instead of a store
    const int po = pl.pad ? n_out : pitch8(n_out), pi = pl.pad ? n_in : pitch8(n_in);
    const bool oi = keep == nullptr || layout == FDP_OUT_IN;     // products that are kept have the output's orientation
    if (!make_rows_map(oi ? &a : &b, G, B, T, pl.planes * po, dt, pitch_g) ||
        !make_rows_map(oi ? &b : &a, X, B, T, pl.planes * pi, dt, pitch_x))
      return FDP_ERR_LAUNCH;
    const int ctas = ctas_per_tile();
    args.M = oi ? n_out : n_in; args.N = oi ? n_in : n_out; args.ld_out = args.N;
    args.tiles_m = ceil_div(args.M, BM * ctas); args.tiles_n = ceil_div(args.N, BN);
    args.tiles_per_batch = args.tiles_m * args.tiles_n;
    args.k_stages = ceil_div(T, BK);
    args.plane_a = oi ? po : pi; args.plane_b = oi ? pi : po;
    args.idesc = make_idesc(dt, true, true, ctas);
    args.segs = 1; args.seg_stages = args.k_stages; args.sub_stages = pl.planes > 1 ? chain_stages(args.seg_stages, pl.planes) : kept_chain(args.seg_stages, pl.pad);
    args.scale = 1.0f; args.nk = NoiseKey{};
    if (pl.planes > 1) { args.zero_status = 0; args.dependent = 1; }     // follows the split kernel, which has cleared the status word
    args.keep = keep;
    if (pl.planes == 3 && keep != nullptr) args.flush_stages = kept_flush(B, args.k_stages, n_in, n_out);
    if (pl.planes == 1)
      return ctas == 2 ? launch<true, true, EPI_CHAIN_SUMSQ, 2>(a, b, a, b, a, args, s)
                       : launch<true, true, EPI_CHAIN_SUMSQ, 1>(a, b, a, b, a, args, s);
    if (pl.planes == 3)
      return ctas == 2 ? launch<true, true, EPI_SPLIT6_SUMSQ, 2>(a, b, a, b, a, args, s)
                       : launch<true, true, EPI_SPLIT6_SUMSQ, 1>(a, b, a, b, a, args, s);
    return ctas == 2 ? launch<true, true, EPI_SPLIT_SUMSQ, 2>(a, b, a, b, a, args, s)
                     : launch<true, true, EPI_SPLIT_SUMSQ, 1>(a, b, a, b, a, args, s);
  }
  if (pl.algo == FDP_NORM_DIRECT) {
    if (!make_rows_map(&a, G, B, T, n_out, dt, pitch_g) || !make_rows_map(&b, X, B, T, n_in, dt, pitch_x)) return FDP_ERR_LAUNCH;
    args.M = n_out; args.N = n_in;
    args.tiles_m = ceil_div(n_out, BM); args.tiles_n = ceil_div(n_in, BN);
    args.tiles_per_batch = args.tiles_m * args.tiles_n;
    args.k_stages = ceil_div(T, BK); args.seg_stages = args.k_stages;
    args.idesc = make_idesc(dt, true, true);
    return launch<true, true, EPI_SUMSQ>(a, b, a, b, a, args, s);
  }
  // A and B boxes are both 128 rows: a B stage is filled by two independent copies
  if (!make_map(&a, G, rows, n_out, BK, BM, dt, pitch_g) || !make_map(&b, G, rows, n_out, BK, BN / 2, dt, pitch_g) ||
      !make_map(&a2, X, rows, n_in, BK, BM, dt, pitch_x) || !make_map(&b2, X, rows, n_in, BK, BN / 2, dt, pitch_x))
    return FDP_ERR_LAUNCH;
  args.M = T; args.N = T;
  args.gram_nb = ceil_div(T, BM);
  args.tiles_m = args.gram_nb; args.tiles_n = args.gram_nb;
  args.tiles_per_batch = gram_tiles(T);
  args.idesc_half = make_idesc(dt, false, false, 1, BN / 2);
  args.k_stages = ceil_div(n_out, BK); args.k_stages2 = ceil_div(n_in, BK);
  args.idesc = make_idesc(dt, false, false);
  return launch<false, false, EPI_GRAM>(a, b, a2, b2, a, args, s);
}

int tc_prescale(const void* G, const float* factors, void* Gs, int B, int T, int n_out, int dt, cudaStream_t s) {
  const size_t nvec = static_cast<size_t>(B) * T * n_out / 8;
  const int vps = T * (n_out / 8);
  const int grid = sm_count() * 8;
  if (dt == FDP_BF16)
    prescale_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>((const __nv_bfloat16*)G, factors, (__nv_bfloat16*)Gs, nvec, vps);
  else
    prescale_kernel<__half><<<grid, 256, 0, s>>>((const __half*)G, factors, (__half*)Gs, nvec, vps);
  note_launch();
  return FDP_OK;
}

static int product_tiles(int M, int N) { return ceil_div(M, BM * ctas_per_tile()) * ceil_div(N, BN); }
int tc_keep_partials(int n_in, int n_out, int layout) {
  return product_tiles(layout == FDP_OUT_IN ? n_out : n_in, layout == FDP_OUT_IN ? n_in : n_out) * ctas_per_tile() * epi_warps_for(EPI_CHAIN_SUMSQ);
}
bool tc_keep_fused_factors_ok(int B, int nparts) { return B <= KEEP_SMEM_FACTORS && B * nparts <= 2048; }
int tc_weighted_sum(const float* keep, const TcFactorSource& fs, void* dW, int B, int n_in, int n_out, int out_dt, int layout,
                    float inv_div, NoiseKey nk, cudaStream_t s, bool wide) {
  const int M = layout == FDP_OUT_IN ? n_out : n_in, N = layout == FDP_OUT_IN ? n_in : n_out;
  const int ctas = ctas_per_tile(), tiles = product_tiles(M, N);
  const int vec_out = N % 4 == 0 && reinterpret_cast<uintptr_t>(dW) % (4 * dtype_size(out_dt)) == 0;
  launch_dependent(wide ? weighted_sum_kernel<true> : weighted_sum_kernel<false>, dim3(tiles * ctas * 32), dim3(256), 0, s, keep, fs, B, ctas, ceil_div(M, BM * ctas),
                   static_cast<size_t>(tiles) * ctas * BM * BN, M, N, dW, out_dt, vec_out, inv_div, nk);
  note_launch();
  return FDP_OK;
}

bool tc_fused_factors_ok(int B) { return B <= MAX_SMEM_FACTORS; }

int tc_clipped_wgrad(const void* Gs, const void* X, const TcFactorSource* fs, float* split_ws,
                     void* dW, int* dev_status, int B, int T, int n_in, int n_out, int dt, int out_dt,
                     int layout, float inv_div, NoiseKey nk, cudaStream_t s, int planes, bool chained, int pitch_g, int pitch_x) {
  const uint64_t rows = static_cast<uint64_t>(B) * T;
  const bool scaled = fs != nullptr;  // Gs is then the unscaled G
  if (planes == 2 && !scaled) return FDP_ERR_ARG;
  CUtensorMap mg, mx, mo, mp;
  // samples are the segments of the K range; a pre-scaled G makes all rows one segment
  const int segs = scaled ? B : 1;
  const uint64_t seg_rows = scaled ? T : rows;
  const int po = planes > 1 ? pitch8(n_out) : n_out, pi = planes > 1 ? pitch8(n_in) : n_in;
  if (!make_rows_map(&mg, Gs, segs, seg_rows, static_cast<uint64_t>(planes) * po, dt, pitch_g) ||
      !make_rows_map(&mx, X, segs, seg_rows, static_cast<uint64_t>(planes) * pi, dt, pitch_x)) return FDP_ERR_LAUNCH;
  TcArgs args{};
  args.batch = 1; args.batch_rows = 0; args.status = dev_status;
  args.dependent = 1;             // always follows a kernel of the same call (norm pass, clip factors or pre-scale)
  args.seg_stages = static_cast<int>((seg_rows + BK - 1) / BK);
  args.k_stages = segs * args.seg_stages;
  args.sub_stages = planes > 1 ? chain_stages(args.seg_stages, planes) : chained ? 1 : args.seg_stages;
  args.out = dW; args.out_dt = out_dt; args.scale = inv_div; args.nk = nk;
  // [out,in]: A = G (M = n_out), B = X (N = n_in); [in,out]: operands swap roles, no transpose pass
  const bool oi = (layout == FDP_OUT_IN);
  args.M = oi ? n_out : n_in; args.N = oi ? n_in : n_out; args.ld_out = args.N;
  const int ctas = ctas_per_tile();
  args.idesc = make_idesc(dt, true, true, ctas);
  if (scaled) {
    args.segs = B;
    args.factors = fs->factors;
    if (fs->factors == nullptr) {
      if (!tc_fused_factors_ok(B) || fs->norm_partials == nullptr) return FDP_ERR_ARG;
      args.norm_partials = fs->norm_partials; args.norm_nparts = fs->nparts;
      args.C = fs->C; args.clamp = fs->clamp;
      args.norms_out = fs->norms_out; args.factors_out = fs->factors_out;
    }
  }
  args.plane_a = oi ? po : pi; args.plane_b = oi ? pi : po;
  args.direct_out = !aligned16(dW) || args.N * dtype_size(out_dt) % 16 != 0;
  args.tiles_m = ceil_div(args.M, BM * ctas); args.tiles_n = ceil_div(args.N, BN);
  args.tiles_per_batch = args.tiles_m * args.tiles_n;
  static const int m_group = [] { const char* e = getenv("FDP_TC_MGROUP"); return e ? atoi(e) : 8; }();
  args.m_group = m_group;
  // tail wave: split K so the SMs left idle by the tile count get work; the parts are parked in the
  // workspace and summed in fixed order by the fix-up kernel (deterministic, no waits)
  const int total = args.tiles_per_batch, workers = launch_sms() / ctas;
  const int split = plan_tail_split(total, args.k_stages, workers, planes == 3 ? 6 : planes == 2 ? 3 : 1);
  // Noise in the epilogue hides behind the main loop of the next tile or of the tile itself (drawn sample by sample).  Where
  // there is one round of short main loops, tiles go to the fix-up kernel as they are and it draws the noise on all SMs:
  // 2 x 71 rows, 576 -> 1472 fp16, 12 tiles of 3 stages, whole call 41 us, parked 21; 5 x 92, 512 -> 512 42 / 20.
  const bool park_whole = nk.std != 0.f && split <= 1 && total <= workers && args.k_stages * (planes == 3 ? 6 : planes == 2 ? 3 : 1) <= 96;
  int n_split_tiles = 0;
  if (split > 1 || park_whole) {
    args.park_whole = park_whole;
    n_split_tiles = total <= workers ? total : total % workers;
    args.split = split;
    args.units_full = total - n_split_tiles;
    args.split_ws = split_ws;
  }
  if (args.direct_out) mo = mg;   // not used
  else if (!make_out_map(&mo, dW, args.M, args.N, out_dt)) return FDP_ERR_LAUNCH;
  // the parked parts: [slot * ctas + CTA of the pair][BM rows][BN columns] fp32
  if (!make_out_map(&mp, split_ws, static_cast<uint64_t>(2) * MAX_SMS * BM, BN, FDP_F32)) return FDP_ERR_LAUNCH;
  int st;
#define FDP_WGRAD_LAUNCH(EPI_, CT_) (oi ? launch<true, true, EPI_, CT_>(mg, mx, mp, mx, mo, args, s) \
                                        : launch<true, true, EPI_, CT_>(mx, mg, mp, mg, mo, args, s))
  if (planes == 3) st = ctas == 2 ? FDP_WGRAD_LAUNCH(EPI_SPLIT6_SCALED, 2) : FDP_WGRAD_LAUNCH(EPI_SPLIT6_SCALED, 1);
  else if (planes == 2) st = ctas == 2 ? FDP_WGRAD_LAUNCH(EPI_SPLIT_SCALED, 2) : FDP_WGRAD_LAUNCH(EPI_SPLIT_SCALED, 1);
  else if (scaled) st = ctas == 2 ? FDP_WGRAD_LAUNCH(EPI_STORE_SCALED, 2) : FDP_WGRAD_LAUNCH(EPI_STORE_SCALED, 1);
  else st = ctas == 2 ? FDP_WGRAD_LAUNCH(EPI_STORE, 2) : FDP_WGRAD_LAUNCH(EPI_STORE, 1);
#undef FDP_WGRAD_LAUNCH
  if (st != FDP_OK || n_split_tiles == 0) return st;
  // the scaled epilogue parks its parts already divided by the batch
  dim3 grid(BM * ctas * BN / (256 * 4), n_split_tiles);
  launch_dependent(splitk_fixup_kernel, grid, dim3(256), 0, s, args.split_ws, args.units_full, split, BM * ctas, args.M,
                   args.N, args.tiles_m, args.tiles_n, args.n_fastest, args.m_group, dW, out_dt, args.ld_out,
                   scaled || planes > 1 ? 1.0f : inv_div, nk, nullptr, 0);
  note_launch();
  return FDP_OK;
}

bool tc_dgrad_ok(int rows, int n_in, int n_out, int dt) {
  return (dt == FDP_BF16 || dt == FDP_F16) && n_in % 8 == 0 && n_out % 8 == 0 && n_in >= 128 && n_out >= 64 && rows >= 128;
}

size_t tc_gemm_park_bytes(int rows, int K, int N, int products) { return gemm_park_bytes(rows, K, N, products); }

// 16-bit products of any width from 64 on.  Operands whose rows are no multiple of 16 bytes are copied first
// (tc_pad_bytes each).  With an fp32 output they took the place of FMA kernels and are to be no further from float64: chained, one
// K stage an accumulator.  Error against float64 and time of FMA kernels / one accumulator for all of K / chained: 8192 rows
// 3648 -> 64 bf16 5.7e-7 312 us / 3.9e-6 15.0 / 1.5e-7 25.0; 5376 rows 5919 -> 320 fp16 1.4e-6 1195 / 7.0e-6 65 / 2.1e-7 81; 1000 rows
// 100 -> 65 6.3e-8 14.7 / 9.8e-8 10.8 / 6.5e-8 10.0.
bool tc_pad_gemm_ok(int rows, int N, int K, int dt) { return (dt == FDP_BF16 || dt == FDP_F16) && rows >= 128 && N >= 64 && K >= 64; }
size_t tc_pad_bytes(size_t rows, int n) { return n % 8 == 0 ? 0 : align256(rows * pitch8(n) * 2); }
int tc_pitch(int n) { return pitch8(n); }

template <bool A_MN, bool B_MN, int EPI>
static int plain_launch(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& a2, const CUtensorMap& b2, const CUtensorMap& o, int ctas,
                        const TcArgs& args, cudaStream_t s) {
  return ctas == 2 ? launch<A_MN, B_MN, EPI, 2>(a, b, a2, b2, o, args, s) : launch<A_MN, B_MN, EPI, 1>(a, b, a2, b2, o, args, s);
}

int tc_dgrad(const void* G, const void* W, void* dX, int* dev_status, int rows, int n_in, int n_out,
             int dt, int out_dt, int w_layout, cudaStream_t s, const GemmPark& park, int pitch_g, int pitch_w, bool chained) {
  CUtensorMap mg, mw, mo;
  const int ctas = ctas_per_tile();
  TcArgs args{};
  args.direct_out = !aligned16(dX) || n_in * dtype_size(out_dt) % 16 != 0;
  if (!make_map(&mg, G, rows, n_out, BK, BM, dt, pitch_g)) return FDP_ERR_LAUNCH;
  if (args.direct_out) mo = mg;   // not used
  else if (!make_out_map(&mo, dX, rows, n_in, out_dt)) return FDP_ERR_LAUNCH;
  args.batch = 1; args.batch_rows = 0; args.status = dev_status; args.zero_status = 1;
  args.M = rows; args.N = n_in; args.ld_out = n_in;
  args.tiles_m = ceil_div(rows, BM * ctas); args.tiles_n = ceil_div(n_in, BN);
  args.tiles_per_batch = args.tiles_m * args.tiles_n;
  args.k_stages = ceil_div(n_out, BK);
  // G is streamed once: CTAs that run together cover a band of rows times all of n_in, so the
  // band of G and the whole of W stay in L2 (walking along M first would re-read G per n-tile)
  args.n_fastest = 1;
  args.out = dX; args.out_dt = out_dt; args.scale = 1.0f; args.nk = NoiseKey{};
  args.segs = 1; args.seg_stages = args.k_stages; args.sub_stages = 1;      // (of a chained product)
  if (w_layout == FDP_OUT_IN) {  // W [n_out, n_in]: rows are K, N contiguous
    if (!make_map(&mw, W, n_out, n_in, 64, BK, dt, pitch_w)) return FDP_ERR_LAUNCH;
    args.idesc = make_idesc(dt, false, true, ctas);
    CUtensorMap mp = mg;
    if (!plan_last_round(args, ctas, make_idesc(dt, false, true, ctas, BN / 2), n_out, 1, park, &mp)) return FDP_ERR_LAUNCH;
    return gemm_fixup(chained ? plain_launch<false, true, EPI_CHAIN_STORE>(mg, mw, mp, mw, mo, ctas, args, s) : plain_launch<false, true, EPI_STORE>(mg, mw, mp, mw, mo, ctas, args, s), args, ctas, s);
  }
  // W [n_in, n_out]: K contiguous; a CTA of a pair loads half of the 256 B rows
  CUtensorMap mh;
  if (!make_map(&mw, W, n_in, n_out, BK, BN / ctas, dt, pitch_w) || !make_map(&mh, W, n_in, n_out, BK, BN / 2 / ctas, dt, pitch_w)) return FDP_ERR_LAUNCH;
  args.idesc = make_idesc(dt, false, false, ctas);
  CUtensorMap mp = mg;
  if (!plan_last_round(args, ctas, make_idesc(dt, false, false, ctas, BN / 2), n_out, 1, park, &mp)) return FDP_ERR_LAUNCH;
  return gemm_fixup(chained ? plain_launch<false, false, EPI_CHAIN_STORE>(mg, mw, mp, mh, mo, ctas, args, s) : plain_launch<false, false, EPI_STORE>(mg, mw, mp, mh, mo, ctas, args, s), args, ctas, s);
}

// forward: A = X [rows, n_in] K-major; B = W, K-major for [n_out, n_in] (Linear), MN-major for
// [n_in, n_out] (Conv1D); bias added in the epilogue
int tc_fwd(const void* X, const void* W, const void* bias, void* Y, int* dev_status, int rows, int n_in,
           int n_out, int dt, int out_dt, int w_layout, cudaStream_t s, const GemmPark& park, int pitch_x, int pitch_w, bool chained) {
  CUtensorMap mx, mw, mo;
  const int ctas = ctas_per_tile();
  TcArgs args{};
  args.direct_out = !aligned16(Y) || n_out * dtype_size(out_dt) % 16 != 0;
  if (!make_map(&mx, X, rows, n_in, BK, BM, dt, pitch_x)) return FDP_ERR_LAUNCH;
  if (args.direct_out) mo = mx;   // not used
  else if (!make_out_map(&mo, Y, rows, n_out, out_dt)) return FDP_ERR_LAUNCH;
  args.batch = 1; args.batch_rows = 0; args.status = dev_status; args.zero_status = 1;
  args.M = rows; args.N = n_out; args.ld_out = n_out;
  args.tiles_m = ceil_div(rows, BM * ctas); args.tiles_n = ceil_div(n_out, BN);
  args.tiles_per_batch = args.tiles_m * args.tiles_n;
  args.k_stages = ceil_div(n_in, BK);
  args.n_fastest = 1;  // X is streamed once, W stays in L2
  args.out = Y; args.out_dt = out_dt; args.scale = 1.0f; args.nk = NoiseKey{};
  args.bias = bias; args.bias_dt = dt; args.bias_vec = aligned16(bias);
  args.segs = 1; args.seg_stages = args.k_stages; args.sub_stages = 1;
  if (w_layout == FDP_OUT_IN) {  // W [n_out, n_in]: K contiguous
    CUtensorMap mh;
    if (!make_map(&mw, W, n_out, n_in, BK, BN / ctas, dt, pitch_w) || !make_map(&mh, W, n_out, n_in, BK, BN / 2 / ctas, dt, pitch_w)) return FDP_ERR_LAUNCH;
    args.idesc = make_idesc(dt, false, false, ctas);
    CUtensorMap mp = mx;
    if (!plan_last_round(args, ctas, make_idesc(dt, false, false, ctas, BN / 2), n_in, 1, park, &mp)) return FDP_ERR_LAUNCH;
    return gemm_fixup(chained ? plain_launch<false, false, EPI_CHAIN_STORE>(mx, mw, mp, mh, mo, ctas, args, s) : plain_launch<false, false, EPI_STORE>(mx, mw, mp, mh, mo, ctas, args, s), args, ctas, s);
  }
  if (!make_map(&mw, W, n_in, n_out, 64, BK, dt, pitch_w)) return FDP_ERR_LAUNCH;  // W [n_in, n_out]: N contiguous
  args.idesc = make_idesc(dt, false, true, ctas);
  CUtensorMap mp = mx;
  if (!plan_last_round(args, ctas, make_idesc(dt, false, true, ctas, BN / 2), n_in, 1, park, &mp)) return FDP_ERR_LAUNCH;
  return gemm_fixup(chained ? plain_launch<false, true, EPI_CHAIN_STORE>(mx, mw, mp, mw, mo, ctas, args, s) : plain_launch<false, true, EPI_STORE>(mx, mw, mp, mw, mo, ctas, args, s), args, ctas, s);
}

// ---- fp32 products on the tensor cores: Y[rows, N] = A[rows, K] * W (+ bias) --------------------------
// A3 is [rows, 2K] and W3 [K, 2N] (w_kn) or [N, 2K] (else): bf16 high halves then low halves (tc_split), or three
// parts each (planes), of which the first two are the halves.
// Three bf16 products per K range into accumulators that the epilogue warps take over every few K
// stages and sum in registers (chain_stages), then the ordinary store epilogue.
bool tc_gemm3_ok(int rows, int K, int N) {
  return rows >= 128 && K >= 128 && N >= 128 && K % BK == 0 && N % 8 == 0;
}
size_t tc_gemm3_w_bytes(int K, int N, int planes) { return align256(static_cast<size_t>(K) * N * 2 * planes); }
size_t tc_gemm3_ws_bytes(int rows, int K, int N) {
  return align256(static_cast<size_t>(rows) * K * 4) + align256(static_cast<size_t>(K) * N * 4);
}
int tc_gemm3(const void* A3, const void* W3, const void* bias, void* Y, int* dev_status, int rows, int K, int N,
             int out_dt, bool w_kn, cudaStream_t s, const GemmPark& park, int planes) {
  CUtensorMap ma, mw, mo;
  const int ctas = ctas_per_tile();
  if (!make_map(&ma, A3, rows, static_cast<uint64_t>(planes) * K, BK, BM, FDP_BF16) || !make_out_map(&mo, Y, rows, N, out_dt)) return FDP_ERR_LAUNCH;
  TcArgs args{};
  args.batch = 1; args.batch_rows = 0; args.status = dev_status;
  args.dependent = 1;            // follows the split kernels of the same call
  args.M = rows; args.N = N; args.ld_out = N;
  args.tiles_m = ceil_div(rows, BM * ctas); args.tiles_n = ceil_div(N, BN);
  args.tiles_per_batch = args.tiles_m * args.tiles_n;
  args.k_stages = K / BK;
  args.plane_a = K; args.plane_b = w_kn ? N : K;
  args.n_fastest = 1;
  args.out = Y; args.out_dt = out_dt; args.scale = 1.0f; args.nk = NoiseKey{};
  args.bias = bias; args.bias_dt = FDP_F32; args.bias_vec = aligned16(bias);
  args.segs = 1; args.seg_stages = args.k_stages; args.sub_stages = chain_stages(args.seg_stages, 2);
  if (w_kn) {   // rows of W3 are K, N contiguous
    if (!make_map(&mw, W3, K, static_cast<uint64_t>(planes) * N, 64, BK, FDP_BF16)) return FDP_ERR_LAUNCH;
    args.idesc = make_idesc(FDP_BF16, false, true, ctas);
    CUtensorMap mp = ma;
    if (!plan_last_round(args, ctas, make_idesc(FDP_BF16, false, true, ctas, BN / 2), K, 3, park, &mp)) return FDP_ERR_LAUNCH;
    return gemm_fixup(ctas == 2 ? launch<false, true, EPI_SPLIT_STORE, 2>(ma, mw, mp, mw, mo, args, s)
                                : launch<false, true, EPI_SPLIT_STORE, 1>(ma, mw, mp, mw, mo, args, s), args, ctas, s);
  }
  CUtensorMap mh;
  if (!make_map(&mw, W3, N, static_cast<uint64_t>(planes) * K, BK, BN / ctas, FDP_BF16) ||                        // K contiguous
      !make_map(&mh, W3, N, static_cast<uint64_t>(planes) * K, BK, BN / 2 / ctas, FDP_BF16)) return FDP_ERR_LAUNCH;
  args.idesc = make_idesc(FDP_BF16, false, false, ctas);
  CUtensorMap mp = ma;
  if (!plan_last_round(args, ctas, make_idesc(FDP_BF16, false, false, ctas, BN / 2), K, 3, park, &mp)) return FDP_ERR_LAUNCH;
  return gemm_fixup(ctas == 2 ? launch<false, false, EPI_SPLIT_STORE, 2>(ma, mw, mp, mh, mo, args, s)
                              : launch<false, false, EPI_SPLIT_STORE, 1>(ma, mw, mp, mh, mo, args, s), args, ctas, s);
}

// The same as six products, for the shapes that three do not take: K and N of any number (the copies' rows are padded,
// their maps end at the last column), an output of any alignment.  These ran on cuBLAS's or this library's fp32 FMA
// kernels and are to be no further from float64.  Against cuBLAS (bias added): 1024 rows 1000 -> 1024 21.9 / 43.1 us, error
// 1.0e-7 / 5.7e-7; 2376 rows 1168 -> 312 27.6 / 54; 5000 rows 900 -> 900 56 / 195; 128 rows 8190 -> 8191 243 / 333; 128 rows
// 1001 -> 4097 26 / 32; 130 rows 72 -> 100 9.6 / 6.1, which is why the Python layer asks for it from 2^26 multiply-adds on.
// Operands that hold an infinity, or what bf16 rounds to one, or nothing but the smallest numbers are done again (simt_redo).
bool tc_gemm6_ok(int rows, int K, int N) {
  constexpr size_t ONE_LAUNCH = static_cast<size_t>(1) << 34;       // elements that tc_split takes at once
  return rows >= 128 && K >= 64 && N >= 64 && static_cast<size_t>(rows) * pitch8(K) < ONE_LAUNCH &&
         static_cast<size_t>(K) * pitch8(N) < ONE_LAUNCH && static_cast<size_t>(N) * pitch8(K) < ONE_LAUNCH;
}
size_t tc_gemm6_w_bytes(int K, int N) {      // in either orientation
  const size_t a = static_cast<size_t>(K) * pitch8(N), b = static_cast<size_t>(N) * pitch8(K);
  return align256((a > b ? a : b) * 6);
}
size_t tc_gemm6_ws_bytes(int rows, int K, int N) {
  return align256(static_cast<size_t>(rows) * pitch8(K) * 6) + SPLIT_MAXIMA_BYTES + tc_gemm6_w_bytes(K, N);
}
int tc_gemm6(const void* A3, const void* W3, const void* bias, void* Y, int* dev_status, int rows, int K, int N,
             int out_dt, bool w_kn, cudaStream_t s, const GemmPark& park) {
  CUtensorMap ma, mw, mh, mo;
  const int ctas = ctas_per_tile();
  TcArgs args{};
  args.direct_out = !aligned16(Y) || N * dtype_size(out_dt) % 16 != 0;
  if (!make_parts_map(&ma, A3, rows, K, BM)) return FDP_ERR_LAUNCH;
  if (args.direct_out) mo = ma;   // not used
  else if (!make_out_map(&mo, Y, rows, N, out_dt)) return FDP_ERR_LAUNCH;
  args.batch = 1; args.batch_rows = 0; args.status = dev_status;
  args.dependent = 1;            // follows the split kernels of the same call
  args.M = rows; args.N = N; args.ld_out = N;
  args.tiles_m = ceil_div(rows, BM * ctas); args.tiles_n = ceil_div(N, BN);
  args.tiles_per_batch = args.tiles_m * args.tiles_n;
  args.k_stages = ceil_div(K, BK);
  args.n_fastest = 1;
  args.out = Y; args.out_dt = out_dt; args.scale = 1.0f; args.nk = NoiseKey{};
  args.bias = bias; args.bias_dt = FDP_F32; args.bias_vec = aligned16(bias);
  args.segs = 1; args.seg_stages = args.k_stages; args.sub_stages = chain_stages(args.seg_stages, 3);
  args.idesc = make_idesc(FDP_BF16, false, w_kn, ctas);
  CUtensorMap mp = ma;
  if (!plan_last_round(args, ctas, make_idesc(FDP_BF16, false, w_kn, ctas, BN / 2), K, 6, park, &mp)) return FDP_ERR_LAUNCH;
  if (w_kn) {   // rows of W3 are K, N contiguous
    if (!make_parts_map(&mw, W3, K, N, BK)) return FDP_ERR_LAUNCH;
    return gemm_fixup(ctas == 2 ? launch<false, true, EPI_SPLIT6_STORE, 2>(ma, mw, mp, mw, mo, args, s)
                                : launch<false, true, EPI_SPLIT6_STORE, 1>(ma, mw, mp, mw, mo, args, s), args, ctas, s);
  }
  if (!make_parts_map(&mw, W3, N, K, BN / ctas) || !make_parts_map(&mh, W3, N, K, BN / 2 / ctas)) return FDP_ERR_LAUNCH;
  return gemm_fixup(ctas == 2 ? launch<false, false, EPI_SPLIT6_STORE, 2>(ma, mw, mp, mh, mo, args, s)
                              : launch<false, false, EPI_SPLIT6_STORE, 1>(ma, mw, mp, mh, mo, args, s), args, ctas, s);
}

}  // namespace fdp
