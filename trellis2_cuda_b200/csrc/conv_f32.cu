// fp32 form of the masked implicit-GEMM sparse conv, on the CUDA cores (the tensor cores would drop the features to tf32).
//
// Operator of src/spconv.cu:91-150 (trellis2-cuda): y[i,co] = sum over taps and input channels of x[nbr[i,v],:] . w[co,v,:],
// fp32 accumulation, absent neighbours contributing zeros.
//
// What bounds it is the FMA rate, once the copies are off the critical path.  One CTA of four warps takes 64 rows of a plan
// tile x 64 output channels and walks the taps that any of ITS rows has (a plan tile's mask covers 128 or 256 rows) in
// chunks of 32 channels through a three-stage ring of cp.async copies, one barrier per chunk.  Both operands lie in shared
// memory as they do in memory (channels innermost, rows 144 bytes apart: the four or eight rows that a warp reads with one
// 16-byte load fall into different banks), and a thread accumulates even and odd channels of its 8 x 4 outputs as pairs
// with fma.rn.f32x2, which needs no operand to be packed or duplicated: 12 shared loads per 64 FMA instructions.
//
// A small map has too few tiles for the 148 SMs (14,534 rows: 228 tiles of 64), so the taps of a tile are split over a
// cluster of S = 4 or 8 CTAs, whose sums meet in distributed shared memory.  S grows until there are three CTAs per SM, as many as
// fit: below that the chip idles, above it the reduction costs more than it gives.  One wave of whole tiles takes about 155 us at
// 64 -> 64 channels however full it is, a wave of quarters 41: from nine tenths of a wave of tiles on S stays 1.
// Every S adds in one order, so a row's bits depend neither on timing nor on the plan nor on how many rows come with it (a scene
// and its parts give the same): tap v belongs to group v % 8, a group is summed by itself, and the eight sums are added in order.
// With S = 1 a CTA adds them up as it goes, with S = 4 it hands on two, with S = 8 one; S = 2 would have to keep four apart.
// Measured, conv alone, 64 -> 64 (without the one order, splits of 1, 2, 4 and 8): 700 rows 25 us (25), 5,000 57 (59), 14,534
// 103 (98), 20,000 129 (121), 60,000 252 (246).
#include "common.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

constexpr int FM = 64, FN = 64, FK = 32, FPITCH = FK + 4, FSTAGES = 3, FTHREADS = 128;
constexpr int F_OPERAND = FM * FPITCH;                          // floats of one operand of one stage (FM == FN)
constexpr int F_SMEM = FSTAGES * 2 * F_OPERAND * (int)sizeof(float);
constexpr int FRED = FN + 4;                                    // row pitch of the groups' sums, which reuse the ring
static_assert(2 * FM * FRED <= FSTAGES * 2 * F_OPERAND, "the sums of two groups fit in the ring");
constexpr int FGROUPS = 8;
constexpr uint32_t FGROUP0 = 0x01010101u;                       // taps of group 0; those of group g are FGROUP0 << g
constexpr uint32_t F_ABSENT = 0x80000000u;

__device__ __forceinline__ void f_copy16(float* dst, const float* src, uint32_t bytes) {       // bytes = 0: zero-fill, src is not read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int S>
__global__ void __launch_bounds__(FTHREADS, 3) k_conv_f32(const float* __restrict__ x, const float* __restrict__ w, const uint32_t* __restrict__ tnbr,
                                                          const int* __restrict__ order, const PlanTile* __restrict__ tiles, const int* __restrict__ perm,
                                                          const int* __restrict__ tile_lo, const int* __restrict__ tile_hi, EpiDev ep,
                                                          float* __restrict__ y, int Ci, int Co, int tile_rows) {
  constexpr int PER = FGROUPS / S, SUMS = S == 1 ? 1 : PER;      // groups of this CTA, and how many sums it hands on
  static_assert(SUMS <= 2, "a CTA of a cluster has one or two groups");
  extern __shared__ __align__(16) float ring[];
  __shared__ uint32_t s_idx[27 * FM];
  __shared__ uint32_t s_mask;
  __shared__ int s_tap[27];
  // consecutive CTAs: the S members of a cluster, then the 64-row parts of a tile, then the tiles (longest first where the plan has perm)
  const int rank = blockIdx.x % S, subs = tile_rows / FM, part = blockIdx.x / S;
  const int pos = *tile_lo + part / subs, sub = part % subs;
  // every CTA of a cluster leaves here or none does: the test does not depend on the rank
  if (pos >= *tile_hi) return;
  const int tile_id = perm ? perm[pos] : pos;
  const PlanTile tile = tiles[tile_id];
  const int rows = min(FM, tile.rows - sub * FM);
  if (rows <= 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, co0 = blockIdx.y * FN;
  const i64 wrow0 = (i64)tile.wbase * Co;

  if (tid == 0) s_mask = 0;
  const uint32_t* tab = tnbr + (i64)tile_id * 27 * tile_rows + sub * FM;
  for (int e = tid; e < 27 * FM; e += FTHREADS) s_idx[e] = __ldg(tab + (e / FM) * tile_rows + e % FM);
  __syncthreads();
  uint32_t have = 0;
  for (int v = warp; v < 27; v += FTHREADS / 32)
    if (__any_sync(0xffffffffu, s_idx[v * FM + lane] != F_ABSENT || s_idx[v * FM + 32 + lane] != F_ABSENT)) have |= 1u << v;
  if (lane == 0 && have) atomicOr(&s_mask, have);
  __syncthreads();
  // this CTA's taps, group by group
  const int g0 = rank * PER;
  const uint32_t mask = s_mask & (FGROUP0 * ((1u << PER) - 1) << g0);
  if (tid < 27 && (mask >> tid & 1))
    s_tap[__popc(mask & FGROUP0 * ((1u << tid % FGROUPS) - 1)) + __popc(mask & FGROUP0 << tid % FGROUPS & ((1u << tid) - 1))] = tid;
  __syncthreads();
  const int nchunk = Ci / FK, steps = __popc(mask) * nchunk;

  // copies: thread t moves 16 bytes of rows t / 8 + 16 i of either operand
  const int l_row = tid >> 3, l_c = (tid & 7) * 4;
  int l_tap = 0, l_chunk = 0, l_stage = 0;            // the next step to be fetched
  auto fetch = [&]() {
    const int v = s_tap[l_tap];
    float* A = ring + l_stage * 2 * F_OPERAND + l_row * FPITCH + l_c;
    float* B = A + F_OPERAND;
    const int k0 = l_chunk * FK + l_c;
#pragma unroll
    for (int i = 0; i < FM / 16; i++) {
      const uint32_t r = s_idx[v * FM + l_row + 16 * i];
      f_copy16(A + 16 * i * FPITCH, x + (i64)(r & 0x7fffffffu) * Ci + k0, r == F_ABSENT ? 0u : 16u);       // absent: row 0, not read
    }
#pragma unroll
    for (int i = 0; i < FN / 16; i++) {
      const int co = co0 + l_row + 16 * i;
      f_copy16(B + 16 * i * FPITCH, w + ((wrow0 + (co < Co ? co : 0)) * 27 + v) * Ci + k0, co < Co ? 16u : 0u);
    }
    if (++l_chunk == nchunk) { l_chunk = 0; l_tap++; }
    if (++l_stage == FSTAGES) l_stage = 0;
  };

  unsigned long long acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
  // outputs of a thread: rows r0 + 4 i, columns c0 + 8 j of the 32 x 32 part of its warp
  const int r0 = (warp >> 1) * 32 + (lane >> 3), c0 = (warp & 1) * 32 + (lane & 7);

#pragma unroll
  for (int s = 0; s < FSTAGES - 1; s++) {
    if (s < steps) fetch();
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float tot[8][4];                         // the sum of the groups before this one (S = 1), or of this CTA's first group
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) tot[i][j] = 0.f;
  int stage = 0, it = 0;
#pragma unroll 1
  for (int g = 0; g < PER; g++) {
    for (const int end = it + __popc(mask & FGROUP0 << (g0 + g)) * nchunk; it < end; it++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
      __syncthreads();                       // this step's copies have landed for everybody, and everybody has read the stage that is filled next
      if (it + FSTAGES - 1 < steps) fetch();
      asm volatile("cp.async.commit_group;" ::: "memory");
      const float* A = ring + stage * 2 * F_OPERAND + r0 * FPITCH;
      const float* B = ring + stage * 2 * F_OPERAND + F_OPERAND + c0 * FPITCH;
#pragma unroll
      for (int k = 0; k < FK; k += 4) {
        ulonglong2 b[4];
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = *(const ulonglong2*)(B + 8 * j * FPITCH + k);
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const ulonglong2 a = *(const ulonglong2*)(A + 4 * i * FPITCH + k);
#pragma unroll
          for (int j = 0; j < 4; j++) { fma2(acc[i][j], a.x, b[j].x); fma2(acc[i][j], a.y, b[j].y); }
        }
      }
      if (++stage == FSTAGES) stage = 0;
    }
    if (S == 1 || g + 1 < PER) {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float2 p = *reinterpret_cast<const float2*>(&acc[i][j]);
          tot[i][j] += p.x + p.y;
          acc[i][j] = 0ull;
        }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // the sums into the ring, then every CTA of the cluster finishes its share of the rows
  float* const red = ring;
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 p = *reinterpret_cast<const float2*>(&acc[i][j]);
      float* const at = red + (r0 + 4 * i) * FRED + c0 + 8 * j;
      if (PER > 1) at[0] = tot[i][j];
      if (S > 1) at[(SUMS - 1) * FM * FRED] = p.x + p.y;
    }
  cg::cluster_group cluster = cg::this_cluster();
  if (S > 1) cluster.sync(); else __syncthreads();
  const float* bias = (const float*)ep.bias; const float* res = (const float*)ep.residual; const float* skx = (const float*)ep.skip_x;
  const int share = FM / S;
  for (int e = tid; e < share * (FN / 4); e += FTHREADS) {
    const int r = rank * share + e / (FN / 4), c = (e % (FN / 4)) * 4, co = co0 + c;
    if (r >= rows || co >= Co) continue;
    float h[4] = {0.f, 0.f, 0.f, 0.f};
    for (int q = 0; q < S; q++) {
      const float* from = S > 1 ? cluster.map_shared_rank(red, q) : red;
#pragma unroll
      for (int k = 0; k < SUMS; k++) {
        const float4 p = *(const float4*)(from + (k * FM + r) * FRED + c);
        h[0] += p.x; h[1] += p.y; h[2] += p.z; h[3] += p.w;
      }
    }
    const int orow = order[tile.start + sub * FM + r];
    int sp = 0, ss = 0;
    if (skx) { const int sv = ep.skip_src[orow]; sp = sv >> 3; ss = sv & 7; }
    const int n = min(4, Co - co);
    float* const yp = y + (i64)orow * Co + co;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (q >= n) break;
      if (bias) h[q] += bias[wrow0 + co + q];
      if (ep.act) h[q] = act_apply(h[q], ep.act);
      if (res) h[q] += res[(i64)orow * Co + co + q];
      if (skx) h[q] += skx[(i64)sp * ep.skip_cin + ss * (ep.skip_cin / 8) + (co + q) / ep.skip_rep];
    }
    if (Co % 4 == 0) *(float4*)yp = make_float4(h[0], h[1], h[2], h[3]);
    else
      for (int q = 0; q < n; q++) yp[q] = h[q];
  }
  if (S > 1) cluster.sync();               // nobody leaves while a peer reads its sums
}

}  // namespace

int conv_f32_launch(t2sc_ctx* ctx, const t2sc_plan* plan, const float* x, const float* w, const EpiDev& ep, float* y, i64 n_in, int Ci, int Co, int part) {
  T2_REQ(ctx, Ci % FK == 0, "Ci=%d", Ci);
  T2_CUDA(ctx, cudaSetDevice(ctx->device));
  const int rc = plan_table_prepare(ctx, const_cast<t2sc_plan*>(plan), n_in);
  if (rc != T2SC_OK) return rc;
  const TilePart tp = tile_part(plan, part);
  const i64 parts = plan->max_tiles * (plan->tile_rows / FM);
  const int ny = cdiv_i(Co, FN);
  const i64 whole = cdiv_i(plan->n_out, FM) * (i64)ny, places = 3ll * ctx->num_sms;
  const int S = 10 * whole >= 9 * places ? 1 : 4 * whole >= places ? 4 : 8;
  const auto kernel = S == 1 ? k_conv_f32<1> : S == 4 ? k_conv_f32<4> : k_conv_f32<8>;
  static bool attr_set[64][9] = {};
  if (ctx->device >= 64 || !attr_set[ctx->device][S]) {
    T2_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM));
    if (ctx->device < 64) attr_set[ctx->device][S] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(parts * S), (unsigned)ny); cfg.blockDim = dim3(FTHREADS); cfg.dynamicSmemBytes = F_SMEM; cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = S > 1 ? 1 : 0;
  T2_CUDA(ctx, cudaLaunchKernelEx(&cfg, kernel, x, w, (const uint32_t*)plan->tnbr, (const int*)plan->order, (const PlanTile*)plan->tiles,
                                  (const int*)(plan->balanced ? plan->perm : nullptr), tp.lo, tp.hi, ep, y, Ci, Co, plan->tile_rows));
  ctx->launches++;
  return T2SC_OK;
}
