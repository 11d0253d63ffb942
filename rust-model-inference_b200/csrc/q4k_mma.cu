// Q4_K matmuls of many activation rows on the tensor cores: the dequantize-and-matmul path and the Q4_K x Q8_K path in
// its exact AVX2 order.  Both use warp-level MMAs (m16n8k16, f32 results in the registers of the threads that scale
// them): the results of two to six MMAs are scaled by per-block factors, so no accumulator could stay in tensor memory
// for longer than that.
//
//   Q4_K x Q8_K (src/ops/quant/mod.rs:701-799).  AVX2 lane L of a super-block sums sc * q * x over 32 values in integers,
//   then acc_L = fma(d_w * d_x, f32(sum), acc_L).  sc * q <= 945 and the bytes x are exact in f16, and a sum of 32 such
//   products is below 2^22, so two m16n8k16 deliver f32(sum) exactly; the eight lanes are eight such pairs on the same
//   operands' other words.  The mins' four chains (mod.rs:749-756) run beside them on exact f32 integers.
//   Bound: no single unit (per warp and super-block of 16 x 16 rows: MMAs 256 cycles of a sub-partition, shared-memory loads
//   400 of the SM, about 400 instructions), at two warps per sub-partition.  11008 x 4096, 200 rows: 116 us (dp4a: 543).
//
//   Dequantize (mod.rs:471-486, tolerance 1e-4): w = (d*sc) * q - dmin*m, so the dot over a 32-block is
//   (d*sc) * sum(q * x) - (dmin*m) * sum(x).  q is exact in bf16 and x is the exact sum of three bf16 values (8 + 8 + 8
//   significant bits), so sum(q * x) is six m16n8k16 with f32 accumulation: no input is rounded.
//   Bound: the MMA rate (8 cycles per 2048 products and sub-partition: 53 us) and the operand loads from shared memory, which
//   take half as long with two weight tiles per warp.  4096 x 4096, 300 rows: 112 us (CUDA cores: 545).
//
// Weights are re-laid out once per path into records whose bytes are in operand-register order (a thread's share of a
// fragment is one aligned piece), activations are written that way by their quantizer / splitter.  The records of the
// weight tiles and of the activation groups of a CTA lie together, K step after K step, so that a stage of its ring is one
// bulk copy of either kind: every further copy costs the issuing warp a few hundred cycles, and with
// one copy per tile the kernels took the sum of their copy and arithmetic times.
#include "common.cuh"
#include "kernels.cuh"
#include "mma_dev.cuh"

namespace {

// ---- record layouts ----
// Q8K weight record, 16 rows x 256 values: [4 pieces][32 threads][16 B] quant words (thread (r, c): row r words L = 0..3,
// L = 4..7 of the 64-value group c, then row r + 8) | [32 threads][8 B] f16 scales (sc[2c], sc[2c+1] of rows r, r + 8) |
// [8][8 B] f16 (d, dmin) of rows r, r + 8 | [16 rows][16 B] f16 mins.
constexpr int Q8K_W = 2624, Q8K_W_SC = 2048, Q8K_W_D = 2304, Q8K_W_MN = 2368;
// Q8K activation record, 8 rows x 256 values: [8 L][32 threads][16 B] f16 | [8 sub-blocks][8 rows] f32 sums | [8] f32 d.
constexpr int Q8K_X = 4384, Q8K_X_S = 4096, Q8K_X_D = 4352;
// Dequantize weight record, 16 rows x 64 values: [32 threads][16 B] quant words (thread (r, c): words 2c, 2c + 1 of row r,
// of row r + 8) | [16 rows] (d*sc, dmin*m of the low sub-block, of the high one) f32.
constexpr int DEQ_W = 768, DEQ_W_S = 512;
// Dequantize activation record, 8 rows x 64 values: [2 sub-blocks][2 words][32 threads][3 pieces x 8 B] bf16 (padded
// order: pieces 0 and 1 as one 16-byte load, piece 2 in a second plane) | [2][8] f32 sums.
constexpr int DEQ_X = 3136, DEQ_X_P2 = 2048, DEQ_X_S = 3072;

struct q4k_params {
  const uint8_t* w;
  const uint8_t* x;
  int steps;            // K in records
  int rt0, rt_end;      // weight row tiles
  int tg_end;           // activation groups
  int tiles_t, n_tiles;
  int m, row_begin, row_end;
  float* out;
  size_t n_rows;
  rmi_dev_status* status;
};

// Weight tiles whose records lie together: those of a CTA.  Of activation groups it is the CTA's number of them, 1 or 2.
constexpr int Q8K_W_PACK = 4, DEQ_W_PACK = 8, X_PACK_MAX = 2;
__host__ __device__ constexpr size_t packed(int pack, size_t i, size_t steps, size_t step) {   // record index
  return (i / pack * steps + step) * pack + i % pack;
}

// RT weight tiles x TG activation groups, KC records of each per stage (several: a stage's barriers and copies take its
// warps a few hundred cycles).
template <int RT, int TG, int WREC, int XREC, int KC, int S>
struct q4k_ring {
  static_assert(S <= 7, "barriers");
  static constexpr int W_STEP = RT * WREC, X_STEP = TG * XREC;
  static constexpr int B0 = KC * W_STEP, STAGE = B0 + KC * X_STEP, SMEM = 128 + S * STAGE;
  int tile, chunk;   // the next item
  __device__ __forceinline__ int blocks(const q4k_params& p) const { return min(KC, p.steps - chunk * KC); }
  __device__ __forceinline__ void copy_w(const q4k_params& p, uint32_t smem, int st) const {
    const size_t tr = p.rt0 / RT + tile / p.tiles_t;
    bulk_load(smem + 128 + st * STAGE, p.w + (tr * p.steps + chunk * KC) * W_STEP, blocks(p) * W_STEP, smem + 8 * st);
  }
  __device__ __forceinline__ void copy_x(const q4k_params& p, uint32_t smem, int st) const {
    const size_t tt = tile % p.tiles_t;
    bulk_load(smem + 128 + st * STAGE + B0, p.x + (tt * p.steps + chunk * KC) * X_STEP, blocks(p) * X_STEP, smem + 8 * st);
  }
  __device__ __forceinline__ void advance(const q4k_params& p) {
    if (++chunk * KC >= p.steps) chunk = 0, tile += gridDim.x;
  }
  // The first S stages, by one thread; the weights' part travels before the wait on the preceding kernel, which writes
  // activations only.
  __device__ __forceinline__ void start(const q4k_params& p, uint32_t smem) {
    for (int pass = 0; pass < 2; pass++) {
      if (pass == 1) pdl_wait();
      tile = blockIdx.x, chunk = 0;
      for (int st = 0; st < S && tile < p.n_tiles; st++) {
        if (pass == 0) {
          mbar_expect_tx(smem + 8 * st, blocks(p) * (W_STEP + X_STEP));
          copy_w(p, smem, st);
        } else {
          copy_x(p, smem, st);
        }
        advance(p);
      }
    }
  }
  __device__ __forceinline__ void next(const q4k_params& p, uint32_t smem, int item, int* abort_flag) {
    if (tile >= p.n_tiles) return;
    const int st = item % S;
    if (!mbar_wait(smem + 64 + 8 * st, ((item / S) & 1) ^ 1, abort_flag, p.status, 15, item)) return;
    mbar_expect_tx(smem + 8 * st, blocks(p) * (W_STEP + X_STEP));
    copy_w(p, smem, st);
    copy_x(p, smem, st);
    advance(p);
  }
};

template <int S>
__device__ __forceinline__ void q4k_ring_init(uint32_t smem, int* abort_flag, int consumers) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < S; i++) {
      mbar_init(smem + 8 * i, 1);
      mbar_init(smem + 64 + 8 * i, consumers);
    }
    *abort_flag = 0;
    mbar_init_fence();
  }
  __syncthreads();
}

__device__ __forceinline__ uint32_t lop_or(uint32_t w, uint32_t mask, uint32_t bits) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(w), "r"(mask), "r"(bits));   // (w & mask) | bits
  return r;
}

// ---------------------------------------------------------------- Q4_K x Q8_K

// Warp tile: 16 weight rows x 8 NG activation rows.
template <int NG, int NWR, int NWT, int KC, int S, int MINB>
__global__ void __launch_bounds__(NWR * NWT * 32, MINB) q4k_q8k_mma_kernel(const q4k_params p) {
  constexpr int RT = NWR, TG = NWT * NG;
  using ring_t = q4k_ring<RT, TG, Q8K_W, Q8K_X, KC, S>;
  static_assert(RT == Q8K_W_PACK && TG <= X_PACK_MAX, "one copy per operand");
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t smem = smem_u32(smem_raw);
  int* abort_flag = reinterpret_cast<int*>(smem_raw + 120);
  q4k_ring_init<S>(smem, abort_flag, NWR * NWT);
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ring_t ring;
  if (threadIdx.x == 0) ring.start(p, smem);
  __syncwarp();
  pdl_wait();
  const int wr = warp / NWT, wt = warp % NWT, r = lane >> 2, c = lane & 3;
  int item = 0;
  for (int tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
    const int tr = tile / p.tiles_t, tt = tile - tr * p.tiles_t;
    const int rt = p.rt0 + tr * RT + wr, t0 = (tt * TG + wt * NG) * 8;
    const bool busy = rt < p.rt_end && t0 < p.m;
    float acc[NG][8][4];
    float accm[NG][4][4];
#pragma unroll
    for (int g = 0; g < NG; g++) {
#pragma unroll
      for (int L = 0; L < 8; L++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[g][L][e] = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; e++)
#pragma unroll
        for (int k = 0; k < 4; k++) accm[g][e][k] = 0.0f;
    }
    for (int ch = 0; ch * KC < p.steps; ch++, item++) {
      const int st = item % S;
      if (!mbar_wait(smem + 8 * st, (item / S) & 1, abort_flag, p.status, 16, item)) return;
      if (threadIdx.x == 0 && item >= 1) ring.next(p, smem, item - 1 + S, abort_flag);
      __syncwarp();
      const int nb = busy ? min(KC, p.steps - ch * KC) : 0;
#pragma unroll 1
      for (int kb = 0; kb < nb; kb++) {
        const uint8_t* wp = smem_raw + 128 + st * ring_t::STAGE + kb * ring_t::W_STEP + wr * Q8K_W;
        const uint8_t* xp = smem_raw + 128 + st * ring_t::STAGE + ring_t::B0 + kb * ring_t::X_STEP + wt * NG * Q8K_X;
        const uint2 scp = *reinterpret_cast<const uint2*>(wp + Q8K_W_SC + lane * 8);
        const uint2 dp = *reinterpret_cast<const uint2*>(wp + Q8K_W_D + r * 8);
        const float2 dd0 = __half22float2(*reinterpret_cast<const __half2*>(&dp.x)), dd1 = __half22float2(*reinterpret_cast<const __half2*>(&dp.y));
        // scale factors of the nibbles as f16 pairs: low (1024 + q) * sc - 1024 sc, high (1024 + 16 q) * sc/16 - 64 sc
        __half2 sl[2], ol[2], sh[2], oh[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const __half2 s2 = *reinterpret_cast<const __half2*>(h ? &scp.y : &scp.x);
          sl[h] = __low2half2(s2);
          sh[h] = __hmul2(__high2half2(s2), __float2half2_rn(0.0625f));
          ol[h] = __hmul2(sl[h], __float2half2_rn(-1024.0f));
          oh[h] = __hmul2(sh[h], __float2half2_rn(-1024.0f));
        }
        float sd[NG][4];
#pragma unroll
        for (int g = 0; g < NG; g++) {
          const float2 dx = *reinterpret_cast<const float2*>(xp + g * Q8K_X + Q8K_X_D + c * 8);
          sd[g][0] = __fmul_rn(dd0.x, dx.x), sd[g][1] = __fmul_rn(dd0.x, dx.y);
          sd[g][2] = __fmul_rn(dd1.x, dx.x), sd[g][3] = __fmul_rn(dd1.x, dx.y);
        }
        // The MMAs of lane L are issued before the results of lane L - 1 are used: an MMA takes about 33 cycles, and
        // consecutive ones have to be independent for the tensor pipe to stay busy.
        float d[2][NG][4];
        uint4 wv[2][2];   // [row half][words 4 h ..]
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int q = 0; q < 2; q++) wv[h][q] = *reinterpret_cast<const uint4*>(wp + h * 1024 + q * 512 + lane * 16);
#pragma unroll
        for (int L = 0; L <= 8; L++) {
          if (L < 8) {
            uint32_t a[2][4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const uint4 w4 = wv[h][L >> 2];
              const uint32_t v = (L & 3) == 0 ? w4.x : ((L & 3) == 1 ? w4.y : ((L & 3) == 2 ? w4.z : w4.w)), v8 = v >> 8;
              const uint32_t t[4] = {lop_or(v, 0x000F000Fu, 0x64006400u), lop_or(v, 0x00F000F0u, 0x64006400u),
                                     lop_or(v8, 0x000F000Fu, 0x64006400u), lop_or(v8, 0x00F000F0u, 0x64006400u)};
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const __half2 y = __hfma2(*reinterpret_cast<const __half2*>(&t[i]), (i & 1) ? sh[h] : sl[h], (i & 1) ? oh[h] : ol[h]);
                a[h][i] = *reinterpret_cast<const uint32_t*>(&y);
              }
            }
            uint4 b[NG];
#pragma unroll
            for (int g = 0; g < NG; g++) b[g] = *reinterpret_cast<const uint4*>(xp + g * Q8K_X + L * 512 + lane * 16);
#pragma unroll
            for (int g = 0; g < NG; g++) mma_f16_k16(d[L & 1][g], a[0][0], a[1][0], a[0][1], a[1][1], b[g].x, b[g].y);
#pragma unroll
            for (int g = 0; g < NG; g++) mma_f16_k16_acc(d[L & 1][g], a[0][2], a[1][2], a[0][3], a[1][3], b[g].z, b[g].w);
          }
          if (L > 0) {
#pragma unroll
            for (int g = 0; g < NG; g++) {
#pragma unroll
              for (int e = 0; e < 4; e++) acc[g][L - 1][e] = __fmaf_rn(sd[g][e], d[(L - 1) & 1][g][e], acc[g][L - 1][e]);   // mod.rs:759-783
            }
          }
        }
        // mins: chain k takes sub-blocks 2k, 2k + 1 (mod.rs:749-756); integers below 2^24, exact in f32
        float mn[2][8];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint4 mv = *reinterpret_cast<const uint4*>(wp + Q8K_W_MN + (r + 8 * h) * 16);
          const uint32_t mw[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&mw[k]));
            mn[h][2 * k] = f.x;
            mn[h][2 * k + 1] = f.y;
          }
        }
#pragma unroll
        for (int g = 0; g < NG; g++) {
          const float2 dx = *reinterpret_cast<const float2*>(xp + g * Q8K_X + Q8K_X_D + c * 8);
          const float dm[4] = {__fmul_rn(-dd0.y, dx.x), __fmul_rn(-dd0.y, dx.y), __fmul_rn(-dd1.y, dx.x), __fmul_rn(-dd1.y, dx.y)};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const float2 sa = *reinterpret_cast<const float2*>(xp + g * Q8K_X + Q8K_X_S + (2 * k) * 32 + c * 8);
            const float2 sc = *reinterpret_cast<const float2*>(xp + g * Q8K_X + Q8K_X_S + (2 * k + 1) * 32 + c * 8);
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const float a0 = (e & 1) ? sa.y : sa.x, a1 = (e & 1) ? sc.y : sc.x;
              const float v = __fmaf_rn(mn[e >> 1][2 * k], a0, __fmul_rn(mn[e >> 1][2 * k + 1], a1));
              accm[g][e][k] = __fmaf_rn(dm[e], v, accm[g][e][k]);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem + 64 + 8 * st);
    }
    if (!busy) continue;
#pragma unroll
    for (int g = 0; g < NG; g++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        float v[8];
#pragma unroll
        for (int L = 0; L < 8; L++) v[L] = acc[g][L][e];
        // hsum_ps (dot.rs:447-456), mins (m0+m2)+(m1+m3) (mod.rs:792-794)
        const float s0 = __fadd_rn(v[4], v[0]), s1 = __fadd_rn(v[5], v[1]), s2v = __fadd_rn(v[6], v[2]), s3 = __fadd_rn(v[7], v[3]);
        const float main_val = __fadd_rn(__fadd_rn(s0, s1), __fadd_rn(s2v, s3));
        const float min_val = __fadd_rn(__fadd_rn(accm[g][e][0], accm[g][e][2]), __fadd_rn(accm[g][e][1], accm[g][e][3]));
        const int row = rt * 16 + r + 8 * (e >> 1), t = t0 + g * 8 + 2 * c + (e & 1);
        if (t < p.m && row >= p.row_begin && row < p.row_end) p.out[(size_t)t * p.n_rows + row] = __fadd_rn(main_val, min_val);
      }
  }
}

// ---------------------------------------------------------------- dequantize

// Warp tile: 16 WR weight rows x 8 NG activation rows.
template <int WR, int NG, int NWR, int NWT, int KC, int S, int MINB>
__global__ void __launch_bounds__(NWR * NWT * 32, MINB) q4k_dequant_mma_kernel(const q4k_params p) {
  constexpr int RT = WR * NWR, TG = NWT * NG;
  using ring_t = q4k_ring<RT, TG, DEQ_W, DEQ_X, KC, S>;
  static_assert(RT == DEQ_W_PACK && TG <= X_PACK_MAX, "one copy per operand");
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t smem = smem_u32(smem_raw);
  int* abort_flag = reinterpret_cast<int*>(smem_raw + 120);
  q4k_ring_init<S>(smem, abort_flag, NWR * NWT);
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ring_t ring;
  if (threadIdx.x == 0) ring.start(p, smem);
  __syncwarp();
  pdl_wait();
  const int wr = warp / NWT, wt = warp % NWT, r = lane >> 2, c = lane & 3;
  const __nv_bfloat162 bias = __float2bfloat162_rn(128.0f);
  int item = 0;
  for (int tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
    const int tr = tile / p.tiles_t, tt = tile - tr * p.tiles_t;
    const int rt = p.rt0 + tr * RT + wr * WR, t0 = (tt * TG + wt * NG) * 8;
    const bool busy = rt < p.rt_end && t0 < p.m;
    float acc[WR][NG][4];
#pragma unroll
    for (int i = 0; i < WR; i++)
#pragma unroll
      for (int g = 0; g < NG; g++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][g][e] = 0.0f;
    for (int ch = 0; ch * KC < p.steps; ch++, item++) {
      const int st = item % S;
      if (!mbar_wait(smem + 8 * st, (item / S) & 1, abort_flag, p.status, 17, item)) return;
      if (threadIdx.x == 0 && item >= 1) ring.next(p, smem, item - 1 + S, abort_flag);
      __syncwarp();
      const int nb = busy ? min(KC, p.steps - ch * KC) : 0;
#pragma unroll 1
      for (int kb = 0; kb < nb; kb++) {
        const uint8_t* wp = smem_raw + 128 + st * ring_t::STAGE + kb * ring_t::W_STEP + wr * WR * DEQ_W;
        const uint8_t* xp = smem_raw + 128 + st * ring_t::STAGE + ring_t::B0 + kb * ring_t::X_STEP + wt * NG * DEQ_X;
        uint4 wq[WR];
        float4 sc[WR][2];
#pragma unroll
        for (int i = 0; i < WR; i++) {
          wq[i] = *reinterpret_cast<const uint4*>(wp + i * DEQ_W + lane * 16);
          sc[i][0] = *reinterpret_cast<const float4*>(wp + i * DEQ_W + DEQ_W_S + r * 16);
          sc[i][1] = *reinterpret_cast<const float4*>(wp + i * DEQ_W + DEQ_W_S + (r + 8) * 16);
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {   // low / high nibbles: the two 32-value sub-blocks
          uint32_t a[WR][2][4];         // [word][r: bytes 0,2 | r+8 | r: bytes 1,3 | r+8]
#pragma unroll
          for (int i = 0; i < WR; i++) {
            const uint32_t wv[2][2] = {{wq[i].x, wq[i].z}, {wq[i].y, wq[i].w}};   // [word][row half]
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
              for (int h = 0; h < 2; h++) {
                const uint32_t v = j ? wv[k][h] >> 4 : wv[k][h];
                const uint32_t t0v = lop_or(v, 0x000F000Fu, 0x43004300u), t1v = lop_or(v >> 8, 0x000F000Fu, 0x43004300u);
                const __nv_bfloat162 y0 = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&t0v), bias);
                const __nv_bfloat162 y1 = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&t1v), bias);
                a[i][k][h] = *reinterpret_cast<const uint32_t*>(&y0);
                a[i][k][2 + h] = *reinterpret_cast<const uint32_t*>(&y1);
              }
          }
          float d[NG][WR][4];
          // consecutive MMAs go to different accumulators: a chain of six on one would take six MMA latencies
#pragma unroll
          for (int k = 0; k < 2; k++) {
            uint4 b[NG];
            uint2 b2[NG];
#pragma unroll
            for (int g = 0; g < NG; g++) {
              b2[g] = *reinterpret_cast<const uint2*>(xp + g * DEQ_X + DEQ_X_P2 + (j * 2 + k) * 256 + lane * 8);
              b[g] = *reinterpret_cast<const uint4*>(xp + g * DEQ_X + (j * 2 + k) * 512 + lane * 16);
            }
#pragma unroll
            for (int piece = 2; piece >= 0; piece--)   // smallest piece first
#pragma unroll
              for (int g = 0; g < NG; g++) {
                const uint32_t b0 = piece == 2 ? b2[g].x : (piece == 1 ? b[g].z : b[g].x);
                const uint32_t b1 = piece == 2 ? b2[g].y : (piece == 1 ? b[g].w : b[g].y);
#pragma unroll
                for (int i = 0; i < WR; i++) {
                  if (k == 0 && piece == 2) mma_bf16_k16(d[g][i], a[i][k][0], a[i][k][1], a[i][k][2], a[i][k][3], b0, b1);
                  else mma_bf16_k16_acc(d[g][i], a[i][k][0], a[i][k][1], a[i][k][2], a[i][k][3], b0, b1);
                }
              }
          }
#pragma unroll
          for (int g = 0; g < NG; g++) {
            const float2 xs = *reinterpret_cast<const float2*>(xp + g * DEQ_X + DEQ_X_S + j * 32 + c * 8);
#pragma unroll
            for (int i = 0; i < WR; i++)
#pragma unroll
              for (int e = 0; e < 4; e++) {
                const float4 f = sc[i][e >> 1];
                const float ds = j ? f.z : f.x, dm = j ? f.w : f.y;
                acc[i][g][e] = __fmaf_rn(-dm, (e & 1) ? xs.y : xs.x, __fmaf_rn(ds, d[g][i][e], acc[i][g][e]));
              }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem + 64 + 8 * st);
    }
    if (!busy) continue;
#pragma unroll
    for (int i = 0; i < WR; i++)
#pragma unroll
      for (int g = 0; g < NG; g++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int row = (rt + i) * 16 + r + 8 * (e >> 1), t = t0 + g * 8 + 2 * c + (e & 1);
          if (t < p.m && row < p.row_end) p.out[(size_t)t * p.n_rows + row] = acc[i][g][e];
        }
  }
}

// ---------------------------------------------------------------- records

__device__ __forceinline__ uint32_t q4k_word(const uint8_t* blk, int g, int wd) {
  return *reinterpret_cast<const uint32_t*>(blk + 16 + 32 * g + 4 * wd);
}
__device__ __forceinline__ int q4k_field(const uint8_t* blk, int j, bool mins) {   // mod.rs:25-33
  const uint8_t* s = blk + 4;
  if (j < 4) return s[j + (mins ? 4 : 0)] & 63;
  return mins ? (s[j + 4] >> 4) | ((s[j] >> 6) << 4) : (s[j + 4] & 15) | ((s[j - 4] >> 6) << 4);
}

// One thread per (row tile, super-block, lane).  Rows past the end repeat the last one.
__global__ void q4k_build_q8k_kernel(const uint8_t* __restrict__ raw, uint8_t* __restrict__ dst, size_t n_rows, size_t n_tiles, size_t nb) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_tiles * nb * 32) return;
  const int lane = (int)(idx & 31), r = lane >> 2, c = lane & 3;
  const size_t sb = (idx >> 5) % nb, tile = (idx >> 5) / nb;
  uint8_t* rec = dst + packed(Q8K_W_PACK, tile, nb, sb) * Q8K_W;
  for (int h = 0; h < 2; h++) {
    const size_t row = min(tile * 16 + r + 8 * h, n_rows - 1);
    const uint8_t* blk = raw + (row * nb + sb) * 144;
    for (int q = 0; q < 2; q++)
      *reinterpret_cast<uint4*>(rec + h * 1024 + q * 512 + lane * 16) =
          make_uint4(q4k_word(blk, c, 4 * q), q4k_word(blk, c, 4 * q + 1), q4k_word(blk, c, 4 * q + 2), q4k_word(blk, c, 4 * q + 3));
    *reinterpret_cast<__half2*>(rec + Q8K_W_SC + lane * 8 + h * 4) =
        __floats2half2_rn((float)q4k_field(blk, 2 * c, false), (float)q4k_field(blk, 2 * c + 1, false));
    *reinterpret_cast<__half2*>(rec + Q8K_W_MN + (r + 8 * h) * 16 + c * 4) =
        __floats2half2_rn((float)q4k_field(blk, 2 * c, true), (float)q4k_field(blk, 2 * c + 1, true));
    if (c == 0) *reinterpret_cast<uint32_t*>(rec + Q8K_W_D + r * 8 + h * 4) = *reinterpret_cast<const uint32_t*>(blk);
  }
}

// One thread per (row tile, 64-value group, lane).
__global__ void q4k_build_deq_kernel(const uint8_t* __restrict__ raw, uint8_t* __restrict__ dst, size_t n_rows, size_t n_tiles, size_t nb) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_tiles * nb * 4 * 32) return;
  const int lane = (int)(idx & 31), r = lane >> 2, c = lane & 3;
  const size_t grp = (idx >> 5) % (nb * 4), tile = (idx >> 5) / (nb * 4);
  const int g = (int)(grp & 3);
  uint8_t* rec = dst + packed(DEQ_W_PACK, tile, nb * 4, grp) * DEQ_W;
  uint32_t w[2][2];
  for (int h = 0; h < 2; h++) {
    const size_t row = min(tile * 16 + r + 8 * h, n_rows - 1);
    const uint8_t* blk = raw + (row * nb + grp / 4) * 144;
    w[h][0] = q4k_word(blk, g, 2 * c);
    w[h][1] = q4k_word(blk, g, 2 * c + 1);
    if (c == 0) {
      const float d = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(blk)), dmin = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(blk + 2));
      *reinterpret_cast<float4*>(rec + DEQ_W_S + (r + 8 * h) * 16) =
          make_float4(__fmul_rn(d, (float)q4k_field(blk, 2 * g, false)), __fmul_rn(dmin, (float)q4k_field(blk, 2 * g, true)),
                      __fmul_rn(d, (float)q4k_field(blk, 2 * g + 1, false)), __fmul_rn(dmin, (float)q4k_field(blk, 2 * g + 1, true)));
    }
  }
  *reinterpret_cast<uint4*>(rec + lane * 16) = make_uint4(w[0][0], w[0][1], w[1][0], w[1][1]);
}

// Q8_K quantizer (mod.rs:82-200) into activation records: one warp per (row, super-block), lane = 8 consecutive values.
__global__ void __launch_bounds__(256) q8k_records_kernel(const float* __restrict__ x, size_t m, size_t nb, int pack,
                                                           uint8_t* __restrict__ dst) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t unit = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  if (unit >= m * nb) return;
  const size_t t = unit / nb, sb = unit - t * nb;
  const float* xp = x + unit * 256 + lane * 8;
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = __ldg(xp + i);
  // first element with the largest |x| (mod.rs:90-97: strict '>' keeps the earliest)
  float best = v[0], ax = fabsf(v[0]);
#pragma unroll
  for (int i = 1; i < 8; i++)
    if (fabsf(v[i]) > ax) ax = fabsf(v[i]), best = v[i];
  int who = lane;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oa = __shfl_xor_sync(0xffffffffu, ax, o), ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int ow = __shfl_xor_sync(0xffffffffu, who, o);
    if (oa > ax || (oa == ax && ow < who)) ax = oa, best = ob, who = ow;
  }
  const float max_val = ax == 0.0f ? 0.0f : best;
  float iscale = 0.0f, dd = 0.0f;
  if (max_val != 0.0f) {
    iscale = __fdiv_rn(-127.0f, max_val);
    dd = __fdiv_rn(1.0f, iscale);
  }
  int q[8], s = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    q[i] = max_val != 0.0f ? max(-127, min(127, (int)rintf(__fmul_rn(v[i], iscale)))) : 0;
    s += q[i];
  }
  const int n = (int)(t & 7);
  uint8_t* rec = dst + packed(pack, t >> 3, nb, sb) * Q8K_X;
  // values 8 lane ..: group c, low / high half, words 2 (lane % 4), + 1
  const int c = lane >> 3, half = (lane >> 2) & 1;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int L = 2 * (lane & 3) + k;
    uint8_t* q16 = rec + L * 512 + (n * 4 + c) * 16 + half * 4;
    *reinterpret_cast<__half2*>(q16) = __floats2half2_rn((float)q[4 * k], (float)q[4 * k + 2]);
    *reinterpret_cast<__half2*>(q16 + 8) = __floats2half2_rn((float)q[4 * k + 1], (float)q[4 * k + 3]);
  }
  // sums of 16 (bsums) wrap to i16, then pairs of them do (mod.rs:749-752): one sum per 32-value sub-block
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  const int bs = (int)(int16_t)s;
  const int pair = (int)(int16_t)(bs + __shfl_xor_sync(0xffffffffu, bs, 2));
  if ((lane & 3) == 0) *reinterpret_cast<float*>(rec + Q8K_X_S + (lane >> 2) * 32 + n * 4) = (float)pair;
  if (lane == 0) *reinterpret_cast<float*>(rec + Q8K_X_D + n * 4) = dd;
}

// x = p0 + p1 + p2 exactly, bf16 each; one warp per (row, 64-value group), lane = 2 consecutive values.
__global__ void __launch_bounds__(256) q4k_split_records_kernel(const float* __restrict__ x, size_t m, size_t groups, int pack,
                                                                 uint8_t* __restrict__ dst) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t unit = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  if (unit >= m * groups) return;
  const size_t t = unit / groups, grp = unit - t * groups;
  const float v[2] = {__ldg(x + unit * 64 + lane * 2), __ldg(x + unit * 64 + lane * 2 + 1)};
  const int n = (int)(t & 7), j = lane >> 4;                 // sub-block
  uint8_t* rec = dst + packed(pack, t >> 3, groups, grp) * DEQ_X;
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int i = (lane & 15) * 2 + u;                       // value inside the sub-block
    const int c = i >> 3, k = (i >> 2) & 1, byte = i & 3;    // thread, word 2 c + k, byte: pairs (0, 2) and (1, 3)
    // rounding towards zero: no piece overflows, and what is left is always representable
    const __nv_bfloat16 p0 = __float2bfloat16_rz(v[u]);
    const float r1 = isfinite(v[u]) ? __fsub_rn(v[u], __bfloat162float(p0)) : 0.0f;
    const __nv_bfloat16 p1 = __float2bfloat16_rz(r1);
    const __nv_bfloat16 p2 = __float2bfloat16_rz(__fsub_rn(r1, __bfloat162float(p1)));
    const int off = (byte & 1) * 4 + (byte >> 1) * 2;
    uint8_t* b = rec + (j * 2 + k) * 512 + (n * 4 + c) * 16 + off;
    *reinterpret_cast<__nv_bfloat16*>(b) = p0;
    *reinterpret_cast<__nv_bfloat16*>(b + 8) = p1;
    *reinterpret_cast<__nv_bfloat16*>(rec + DEQ_X_P2 + (j * 2 + k) * 256 + (n * 4 + c) * 8 + off) = p2;
  }
  double s = (double)v[0] + (double)v[1];
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((lane & 15) == 0) *reinterpret_cast<float*>(rec + DEQ_X_S + j * 32 + n * 4) = (float)s;
}

// ---------------------------------------------------------------- launches

constexpr int Q4K_MAX_DEVICES = 16;

template <typename K>
int32_t q4k_mma_launch(rmi_ctx* ctx, K kern, int* cache, int threads, size_t smem, q4k_params& p, int rt_per_tile, int tg_per_tile,
                       const char* what) {
  int& per_sm = cache[ctx->device % Q4K_MAX_DEVICES];
  if (per_sm == 0) {   // once per kernel and device
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    if (e != cudaSuccess || per_sm < 1) {
      rmi_set_error("%s needs %zu B of shared memory: %s", what, smem, cudaGetErrorString(e));
      return RMI_ERR_CUDA;
    }
  }
  p.tiles_t = (p.tg_end + tg_per_tile - 1) / tg_per_tile;
  p.n_tiles = (p.rt_end - p.rt0 + rt_per_tile - 1) / rt_per_tile * p.tiles_t;
  const int slots = ctx->sm_count * per_sm;
  return rmi_run(ctx, what, kern, dim3((unsigned)(p.n_tiles < slots ? p.n_tiles : slots)), dim3((unsigned)threads), smem, p);
}

template <int NG, int NWR, int NWT, int KC, int S, int MINB>
int32_t run_q8k(rmi_ctx* ctx, q4k_params p) {
  static int cache[Q4K_MAX_DEVICES];
  return q4k_mma_launch(ctx, q4k_q8k_mma_kernel<NG, NWR, NWT, KC, S, MINB>, cache, NWR * NWT * 32,
                        q4k_ring<NWR, NWT * NG, Q8K_W, Q8K_X, KC, S>::SMEM, p, NWR, NWT * NG, "q4k_q8k_mma");
}
template <int WR, int NG, int NWR, int NWT, int KC, int S, int MINB>
int32_t run_deq(rmi_ctx* ctx, q4k_params p) {
  static int cache[Q4K_MAX_DEVICES];
  return q4k_mma_launch(ctx, q4k_dequant_mma_kernel<WR, NG, NWR, NWT, KC, S, MINB>, cache, NWR * NWT * 32,
                        q4k_ring<WR * NWR, NWT * NG, DEQ_W, DEQ_X, KC, S>::SMEM, p, WR * NWR, NWT * NG, "q4k_dequant_mma");
}

int32_t build_records(rmi_ctx* ctx, rmi_weight* w, bool deq) {
  const size_t nb = w->n_in / 256, pack = deq ? DEQ_W_PACK : Q8K_W_PACK;
  const size_t n_tiles = (w->n_tiles16 + pack - 1) / pack * pack, recs = n_tiles * nb * (deq ? 4 : 1);
  const size_t bytes = recs * (deq ? DEQ_W : Q8K_W);
  uint8_t* d = nullptr;
  if (cudaMalloc((void**)&d, bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    return RMI_ERR_OOM;
  }
  const unsigned grid = (unsigned)((recs * 32 + 255) / 256);
  if (deq) q4k_build_deq_kernel<<<grid, 256, 0, ctx->stream>>>(w->d_raw, d, w->n_rows, n_tiles, nb);
  else q4k_build_q8k_kernel<<<grid, 256, 0, ctx->stream>>>(w->d_raw, d, w->n_rows, n_tiles, nb);
  // complete before any kernel of a dependent launch may fetch it ahead of its wait
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
    cudaFree(d);
    return RMI_ERR_CUDA;
  }
  (deq ? w->d_q4k_deq : w->d_q4k_q8k) = d;
  w->frag_bytes += bytes;
  return RMI_OK;
}

q4k_params base_params(rmi_ctx* ctx, const rmi_weight* w, const uint8_t* x, size_t m, float* out) {
  q4k_params p = {};
  p.x = x;
  p.rt_end = (int)w->n_tiles16;
  p.tg_end = (int)((m + 7) / 8);
  p.m = (int)m;
  p.row_end = (int)w->n_rows;
  p.out = out;
  p.n_rows = w->n_rows;
  p.status = ctx->d_status;
  return p;
}

}  // namespace

// The records are built on first use.  False inside a stream capture, or without memory for them.
bool q4k_mma_prepare(rmi_ctx* ctx, const rmi_weight* w, bool dequant) {
  if ((dequant ? w->d_q4k_deq : w->d_q4k_q8k) != nullptr) return true;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    (void)cudaGetLastError();
    return false;
  }
  return build_records(ctx, const_cast<rmi_weight*>(w), dequant) == RMI_OK;
}

size_t q4k_mma_x_bytes(const rmi_weight* w, size_t m, bool dequant) {
  const size_t nb = w->n_in / 256, groups = (m + 8 * X_PACK_MAX - 1) / (8 * X_PACK_MAX) * X_PACK_MAX;
  return dequant ? groups * nb * 4 * DEQ_X : groups * nb * Q8K_X;
}

// AVX2 order; q4k_mma_prepare succeeded; x f32 rows, xrec scratch of q4k_mma_x_bytes
int32_t launch_q4k_q8k_mma(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, uint8_t* xrec, float* out, size_t row_begin,
                           size_t row_end) {
  if (m == 0 || row_begin >= row_end) return RMI_OK;
  // 16 activation rows per CTA (the conversion of the nibbles is shared by two MMA column tiles); 8 where that leaves half
  // of the SMs without work (16 rows of 4096 x 4096: 12.0 -> 7.8 us)
  const size_t packs = (row_end + 16 * Q8K_W_PACK - 1) / (16 * Q8K_W_PACK) - row_begin / (16 * Q8K_W_PACK);
  const int groups = packs * ((m + 15) / 16) * 2 <= (size_t)ctx->sm_count ? 1 : 2;
  const size_t nb = w->n_in / 256, warps = m * nb;
  RMI_TRY(rmi_run(ctx, "q8k_records", q8k_records_kernel, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, x, m, nb, groups, xrec));
  q4k_params p = base_params(ctx, w, xrec, m, out);
  p.w = w->d_q4k_q8k;
  p.steps = (int)nb;
  p.rt0 = (int)(row_begin / (16 * Q8K_W_PACK)) * Q8K_W_PACK;
  p.rt_end = (int)((row_end + 15) / 16);
  p.row_begin = (int)row_begin;
  p.row_end = (int)row_end;
  return groups == 1 ? run_q8k<1, 4, 1, 4, 2, 3>(ctx, p) : run_q8k<2, 4, 1, 3, 2, 2>(ctx, p);
}

int32_t launch_q4k_dequant_mma(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, uint8_t* xrec, float* out) {
  if (m == 0 || w->n_rows == 0) return RMI_OK;
  // 16 activation rows per CTA, 8 while that leaves SMs without work (16 rows of 4096 x 4096: 28.9 -> 22.6 us, 48: 43 -> 36)
  const int tg = (w->n_tiles16 + DEQ_W_PACK - 1) / DEQ_W_PACK * ((m + 15) / 16) <= (size_t)ctx->sm_count ? 1 : 2;
  const size_t groups = w->n_in / 64, warps = m * groups;
  RMI_TRY(rmi_run(ctx, "q4k_split_records", q4k_split_records_kernel, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, x, m, groups, tg, xrec));
  q4k_params p = base_params(ctx, w, xrec, m, out);
  p.w = w->d_q4k_deq;
  p.steps = (int)groups;
  return tg == 1 ? run_deq<2, 1, 4, 1, 4, 2, 3>(ctx, p) : run_deq<2, 2, 4, 1, 4, 2, 2>(ctx, p);
}
