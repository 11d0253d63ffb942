// Batched prompt processing for the Qwen3 session.
//
// The reference feeds the prompt one position at a time (src/models/qwen3.rs:657-689); every operator of a
// step works on one row, and the only coupling between positions is the K/V cache that attention reads.  So
// the prompt positions 0..P-1 of a sequence can run as P rows through each operator -- the matmuls as
// M = P calls of the same per-row kernels (src/ops/kernel/trait_.rs:78-109 defines an M-row matmul as exactly
// that loop), attention causally per position over the cache rows written by the same launch sequence -- and
// every value (cache rows, hidden state) carries the bits the token loop would have produced.  Only the
// position P = n_prompt-1, whose logits are needed, then runs through the regular decode step.
//
// Kernels here: embedding rows, rms_norm rows (f32 out), per-head q/k norm + rotation + cache append for all
// rows, and causal attention for many query positions.  Their arithmetic restates the same reference code as
// the decode-step kernels (paths inside the reference project):
//   rms_norm       src/ops/norm.rs:3-19           f32 squares summed in f64
//   rope / cache   src/ops/rope.rs:21-37, src/models/qwen3.rs:851-870
//   attention      src/models/qwen3.rs:876-933    f16 q/k/v/p, sequential f64 dots (src/ops/dot.rs:99-119),
//                                                 softmax with the sequential f32 sum (src/ops/attention.rs:28-38)
#include "common.cuh"
#include "decode.cuh"
#include "decode_dev.cuh"
#include "kernels.cuh"

namespace {

// x[r][:] = f16(d) * q of row prompts[b][p]; r = b_local * P + p
__global__ void embed_rows_kernel(const uint8_t* __restrict__ emb, size_t blocks, const uint32_t* __restrict__ prompts,
                                  size_t n_prompt, size_t P, size_t b0, float* __restrict__ x, uint32_t vocab) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t r = blockIdx.x, b = b0 + r / P, p = r % P;
  uint32_t tok = prompts[b * n_prompt + p];
  if (tok >= vocab) tok = 0;  // rejected on the host before the first launch
  const uint8_t* base = emb + (size_t)(tok / 16) * blocks * Q8_REC_BYTES;
  const int rr = tok % 16;
  for (size_t i = threadIdx.x; i < blocks * 32; i += blockDim.x) {
    const uint8_t* rec = base + (i / 32) * Q8_REC_BYTES;
    const float d = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(rec + 2 * rr));
    x[r * blocks * 32 + i] = __fmul_rn(d, (float)(int8_t)rec[32 + 32 * rr + (i & 31)]);
  }
}

// x += add (optional); out = rms_norm(x) * weight.  One CTA of 256 threads per row.
__global__ void rmsnorm_rows_kernel(float* __restrict__ x, const float* __restrict__ add, const float* __restrict__ weight,
                                    size_t n, float eps, float* __restrict__ out) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ double s_part[8];
  __shared__ float s_scale;
  const size_t r = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* xr = x + r * n;
  double part = 0.0;
  for (size_t i = threadIdx.x; i < n; i += blockDim.x) {
    float v = xr[i];
    if (add) {
      v = __fadd_rn(v, add[r * n + i]);
      xr[i] = v;
    }
    part += (double)__fmul_rn(v, v);
  }
  part = warp_sum_f64(part);
  if (lane == 0) s_part[warp] = part;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 8; w++) s += s_part[w];
    const float mean_sq = (float)(s / (double)n);
    s_scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean_sq, eps)));
  }
  __syncthreads();
  const float sc = s_scale;
  for (size_t i = threadIdx.x; i < n; i += blockDim.x) out[r * n + i] = __fmul_rn(__fmul_rn(xr[i], sc), weight[i]);
}

// One warp per (row, head), eight per CTA (CTAs of one warp: 18 us for 479 rows of 32 heads, 102 for 3040;
// here 31 for 3040): q -> q16[r], k/v -> cache row (b, layer, p)
__global__ void qk_norm_rope_kv_rows_kernel(const float* __restrict__ qkv, size_t n_head, size_t n_head_kv, size_t hd,
                                            const float* __restrict__ q_norm, const float* __restrict__ k_norm, float eps,
                                            const float* __restrict__ rope, size_t P, size_t b0,
                                            uint16_t* __restrict__ q16, uint16_t* __restrict__ k_cache,
                                            uint16_t* __restrict__ v_cache, size_t layer, size_t n_layer, size_t capacity, size_t rows) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t heads = n_head + 2 * n_head_kv, unit = (size_t)blockIdx.x * 8 + threadIdx.x / 32;
  const size_t r = unit / heads, head = unit - r * heads, b = b0 + r / P, p = r % P;
  const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  const size_t nq = n_head * hd, nk = n_head_kv * hd;
  const float* src = qkv + r * (nq + 2 * nk) + head * hd;
  const size_t cache_row = ((b * n_layer + layer) * capacity + p) * nk;
  if (head >= n_head + n_head_kv) {  // V: straight f16 conversion
    const size_t kvh = head - n_head - n_head_kv;
    for (size_t i = lane; i < hd; i += 32) v_cache[cache_row + kvh * hd + i] = f32_to_f16_bits(src[i]);
    return;
  }
  const bool is_q = head < n_head;
  uint16_t* dst = is_q ? q16 + r * nq + head * hd : k_cache + cache_row + (head - n_head) * hd;
  norm_rope_head_f16(src, is_q ? q_norm : k_norm, eps, rope + p * hd, hd, lane, dst);
}

// Causal attention of up to eight query rows of one (sequence, kv head); row r of a kv head is query head r % group of the
// group that shares it, at position r / group, so a CTA's rows are consecutive positions.  Per row the arithmetic is that
// of one decode step: sequential f64 dot over the head dimension, f32 score * 1/sqrt(hd), max, exp, sequential f32 sum over
// the positions, divide, f16, then per output element the f64 sum over the positions in ascending order.
//
// Bound: the f64 pipe, two multiply-adds per query row, visible position and head element (a conversion to f64 takes four
// times as long as a multiply-add, so the products are not converted).  A product of two f16 values is exact, so a fused
// multiply-add rounds as a multiplication and an addition would, and m8n8k4 f64 MMAs add their four products one after the
// other in ascending order, each with one rounding (checked against chains of fma on operands of full precision: no bit
// differs).  Multiply-add instructions of the CUDA cores run at 2.7 cycles instead of 2 on three 64-bit register operands
// and need a load per four of them; an MMA is 16 cycles for 256 multiply-adds and one value per thread and operand.
// Measured, 16 query and 8 kv heads of 128: 480 positions 225 -> 64 us, 960 positions 209 us (the MMAs alone: 26 and 104 us;
// the rest is the soft-max, the f16 conversions and the staging of K and V, which four CTAs per SM overlap in part).
// f16 -> f64 in integer instructions: of the f64 form only the high word is not zero, and with the exponent left 1008 too
// small (2^1008 is put into the other factor; both exact) that word is the sign-extended f16 shifted and masked.
constexpr int PF_THREADS = 128, PF_TILE = 64;

__device__ __forceinline__ double f16_small_f64(int16_t bits) {   // x * 2^-1008 of the f16 value x, infinities and NaNs too
  const int h = bits;
  int hi = (int)(((uint32_t)h << 10) & 0x81ffffffu);
  if ((~h & 0x7c00) == 0) hi |= 0x7ff00000;
  return __hiloint2double(hi, 0);
}
__device__ __forceinline__ int f32_hi_large(float v) {          // high word of v * 2^1008 for f16-valued v; the low one is 0
  return __double2hiint((double)v * 0x1p1008);
}
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

// Four warps.  Scores: a warp takes every fourth 8-position tile, its rows of Q stay in registers.  Outputs: a warp takes
// HD / 4 head elements.  K and V tiles of 64 positions stream through two buffers.
template <int HD>
__global__ void __launch_bounds__(PF_THREADS, 3)
    attention_prefill_kernel(const uint16_t* __restrict__ q16, const uint16_t* __restrict__ k_cache,
                             const uint16_t* __restrict__ v_cache, size_t n_head, size_t n_head_kv, size_t layer,
                             size_t n_layer, size_t capacity, size_t P, size_t b0, size_t n_seq, int rows_per_cta,
                             float* __restrict__ attn_out) {
  constexpr int STRIDE = HD + 8, TILE = PF_TILE * STRIDE, NT = HD / 32;   // f16 row stride: rows four banks apart
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t pf_smem[];
  int16_t* kv = reinterpret_cast<int16_t*>(pf_smem);               // 2 x [PF_TILE][STRIDE]
  int* sc = reinterpret_cast<int*>(pf_smem + 2 * TILE * 2);         // [rows][cs] scores, exponentials (f32), high words of p * 2^1008
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
  // the longest rows of every head and sequence start first, the shortest fill the gaps at the end
  const size_t kvh = blockIdx.x % n_head_kv, bl = blockIdx.x / n_head_kv % n_seq, b = b0 + bl;
  const int group = (int)(n_head / n_head_kv);
  const int r0 = (int)((gridDim.x - 1 - blockIdx.x) / (n_head_kv * n_seq)) * rows_per_cta;
  const int rows = min(rows_per_cta, (int)P * group - r0);
  const int T = (r0 + rows - 1) / group + 1;                         // cache positions that any row may see
  const int n_tiles = (T + PF_TILE - 1) / PF_TILE, cs = n_tiles * PF_TILE + 4;
  const size_t nq = n_head * HD, nk = n_head_kv * HD;
  const float kq_scale = __fdiv_rn(1.0f, __fsqrt_rn((float)HD));
  const uint16_t* kbase = k_cache + ((b * n_layer + layer) * capacity) * nk + kvh * HD;
  const uint16_t* vbase = v_cache + ((b * n_layer + layer) * capacity) * nk + kvh * HD;
  auto stage = [&](const uint16_t* base, int tile) {   // positions past T repeat the last one
    int16_t* dst = kv + (tile & 1) * TILE;
#pragma unroll
    for (int u = 0; u < PF_TILE * HD / 8 / PF_THREADS; u++) {
      const int i = tid + PF_THREADS * u, t = min(tile * PF_TILE + i / (HD / 8), T - 1);
      cp_async16(dst + i / (HD / 8) * STRIDE + i % (HD / 8) * 8, base + (size_t)t * nk + i % (HD / 8) * 8);
    }
    cp_async_commit();
  };
  auto arrived = [&](bool more) {
    if (more) cp_async_wait<1>(); else cp_async_wait<0>();
    __syncthreads();
  };
  stage(kbase, 0);
  const int fr = r0 + min(r, rows - 1), pos = r < rows ? fr / group : -1;   // this thread's row and its position
  const size_t row_off = (bl * P + fr / group) * nq + (kvh * group + fr % group) * HD;

  // scores[row][t] = f32(sum_f64 q*k) * kq_scale for t <= position of the row (dot.rs:115-118)
  {
    int qh[HD / 4];
#pragma unroll
    for (int s = 0; s < HD / 4; s++) qh[s] = f32_hi_large(f16_bits_to_f32(q16[row_off + 4 * s + c]));
    for (int tile = 0; tile < n_tiles; tile++) {
      if (tile + 1 < n_tiles) stage(kbase, tile + 1);
      arrived(tile + 1 < n_tiles);
      const int16_t* kt = kv + (tile & 1) * TILE + (8 * warp + r) * STRIDE + c;
      const int t0 = tile * PF_TILE + 8 * warp;   // this warp: positions t0 .. t0 + 7 and t0 + 32 .. t0 + 39
      if (t0 < T) {
        double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
        for (int s = 0; s < HD / 4; s++) {
#pragma unroll
          for (int n = 0; n < 2; n++) mma_f64(acc[n], __hiloint2double(qh[s], 0), f16_small_f64(kt[32 * n * STRIDE + 4 * s]));
        }
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int t = t0 + 32 * n + 2 * c + e;
            if (t <= pos) sc[r * cs + t] = __float_as_int(__fmul_rn((float)acc[n][e], kq_scale));
          }
      }
      __syncthreads();
    }
  }

  stage(vbase, 0);  // the first V tile travels while the soft-max is evaluated
  // per row: max, exp, sequential f32 sum (attention.rs:28-38), divide, f16
  for (int row = warp; row < rows; row += 4) {
    const int Tr = (r0 + row) / group + 1;
    float* e = reinterpret_cast<float*>(sc + row * cs);
    float mx = -INFINITY;
    for (int t = lane; t < Tr; t += 32) mx = fmaxf(mx, e[t]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll 2
    for (int t = lane; t < Tr; t += 32) e[t] = exp_cr(__fsub_rn(e[t], mx));
  }
  __syncwarp();
  float sum = 0.0f;   // lane i: the warp's row i
  if (warp + 4 * lane < rows) {
    const int row = warp + 4 * lane, Tr = (r0 + row) / group + 1;
    const float* e = reinterpret_cast<const float*>(sc + row * cs);
    int t = 0;
#pragma unroll 4
    for (; t + 4 <= Tr; t += 4) {
      const float4 v = *reinterpret_cast<const float4*>(e + t);
      sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v.x), v.y), v.z), v.w);
    }
    for (; t < Tr; t++) sum = __fadd_rn(sum, e[t]);
  }
  for (int row = warp, i = 0; row < rows; row += 4, i++) {
    const int Tr = (r0 + row) / group + 1;
    const float s = __shfl_sync(0xffffffffu, sum, i);
    int* e = sc + row * cs;
    for (int t = lane; t < Tr; t += 32) {
      float pv = __int_as_float(e[t]);
      if (s > 0.0f) pv = __fdiv_rn(pv, s);
      e[t] = f32_hi_large(f16_bits_to_f32(f32_to_f16_bits(pv)));
    }
  }

  // out[row][d] = f32(sum_f64 over t ascending of v[t][d] * p[row][t]): MMAs over the positions that every row sees (a
  // multiple of four), the few after them one by one for the rows that see them
  const int t_all = (r0 / group + 1) & ~3;
  double acc[NT][2];
#pragma unroll
  for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = 0.0;
  const int d0 = warp * (HD / 4);
  const int* prow = sc + min(r, rows - 1) * cs;
  for (int tile = 0; tile < n_tiles; tile++) {
    if (tile + 1 < n_tiles) stage(vbase, tile + 1);
    arrived(tile + 1 < n_tiles);
    const int16_t* vt = kv + (tile & 1) * TILE + d0;
    const int t0 = tile * PF_TILE, full = min(PF_TILE, t_all - t0), nt = min(PF_TILE, T - t0);
#pragma unroll 4
    for (int t = 0; t < full; t += 4) {
      const double p = __hiloint2double(prow[t0 + t + c], 0);
#pragma unroll
      for (int n = 0; n < NT; n++) mma_f64(acc[n], p, f16_small_f64(vt[(t + c) * STRIDE + 8 * n + r]));
    }
    for (int t = max(full, 0); t < nt && t0 + t <= pos; t++) {
      const double p = __hiloint2double(prow[t0 + t], 0);
#pragma unroll
      for (int n = 0; n < NT; n++) {
        const uint32_t v2 = *reinterpret_cast<const uint32_t*>(vt + t * STRIDE + 8 * n + 2 * c);
        acc[n][0] = __fma_rn(f16_small_f64((int16_t)(v2 & 0xffffu)), p, acc[n][0]);
        acc[n][1] = __fma_rn(f16_small_f64((int16_t)(v2 >> 16)), p, acc[n][1]);
      }
    }
    __syncthreads();
  }
  if (r < rows) {
    float* o = attn_out + row_off + d0 + 2 * c;
#pragma unroll
    for (int n = 0; n < NT; n++) *reinterpret_cast<float2*>(o + 8 * n) = make_float2((float)acc[n][0], (float)acc[n][1]);
  }
}

__global__ void set_step_kernel(int* d_step, int value) {
  pdl_wait();
  pdl_launch_dependents();
  *d_step = value;
}

size_t prefill_attention_smem(int rows, size_t P, size_t hd) {
  const size_t cs = (P + PF_TILE - 1) / PF_TILE * PF_TILE + 4;
  return 2 * PF_TILE * (hd + 8) * 2 + rows * cs * 4;
}

}  // namespace

// Query rows per CTA: the eight of an MMA row tile, fewer only where the scores of a long prompt leave no room.  0: none.
// Sixteen rows (two row tiles share the conversion of K and V) are no faster: half as many CTAs even out less well.
int prefill_attention_rows(const rmi_ctx* ctx, const decode_dims& d, size_t P) {
  for (int rows = 8; rows >= 1; rows >>= 1)
    if (prefill_attention_smem(rows, P, d.hd) <= ctx->smem_optin) return rows;
  return 0;
}

bool prefill_supported(const rmi_ctx* ctx, const decode_dims& d, size_t P) {
  return (d.hd == 128 || d.hd == 64 || d.hd == 32) && d.n_head % d.n_head_kv == 0 && prefill_attention_rows(ctx, d, P) > 0;
}

int32_t launch_embed_rows(rmi_ctx* ctx, const rmi_weight* emb, const uint32_t* prompts, size_t n_prompt, size_t P, size_t b0,
                          size_t rows, float* x) {
  return rmi_run(ctx, "embed_rows", embed_rows_kernel, dim3((unsigned)rows), dim3(256), 0, emb->d_tile16, emb->n_in / 32, prompts,
                 n_prompt, P, b0, x, (uint32_t)emb->n_rows);
}

int32_t launch_rmsnorm_rows(rmi_ctx* ctx, float* x, const float* add, const float* weight, size_t n, float eps, float* out,
                            size_t rows) {
  return rmi_run(ctx, "rmsnorm_rows", rmsnorm_rows_kernel, dim3((unsigned)rows), dim3(256), 0, x, add, weight, n, eps, out);
}

int32_t launch_qk_norm_rope_kv_rows(rmi_ctx* ctx, const decode_dims& d, const float* qkv, const float* q_norm,
                                    const float* k_norm, const float* rope, size_t P, size_t b0, size_t rows, uint16_t* q16,
                                    uint16_t* k_cache, uint16_t* v_cache, size_t layer) {
  const dim3 grid((unsigned)((rows * (d.n_head + 2 * d.n_head_kv) + 7) / 8));
  return rmi_run(ctx, "qk_norm_rope_kv_rows", qk_norm_rope_kv_rows_kernel, grid, dim3(256), 0, qkv, d.n_head, d.n_head_kv, d.hd, q_norm,
                 k_norm, d.eps, rope, P, b0, q16, k_cache, v_cache, layer, d.n_layer, d.capacity, rows);
}

int32_t launch_attention_prefill(rmi_ctx* ctx, const decode_dims& d, const uint16_t* q16, const uint16_t* k_cache,
                                 const uint16_t* v_cache, size_t layer, size_t P, size_t b0, size_t n_seq, float* attn_out) {
  const int rows = prefill_attention_rows(ctx, d, P);
  RMI_REQUIRE(rows > 0, RMI_ERR_UNSUPPORTED, "prompt of %zu positions does not fit the prefill attention kernel", P);
  const size_t group = d.n_head / d.n_head_kv, smem = prefill_attention_smem(rows, P, d.hd);
  auto kern = d.hd == 128 ? attention_prefill_kernel<128> : (d.hd == 64 ? attention_prefill_kernel<64> : attention_prefill_kernel<32>);
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    (void)cudaGetLastError();
    rmi_set_error("prefill attention needs %zu B of shared memory", smem);
    return RMI_ERR_UNSUPPORTED;
  }
  const size_t grid = (P * group + rows - 1) / rows * d.n_head_kv * n_seq;
  return rmi_run(ctx, "attention_prefill", kern, dim3((unsigned)grid), dim3(PF_THREADS), smem, q16, k_cache, v_cache, d.n_head, d.n_head_kv, layer,
                 d.n_layer, d.capacity, P, b0, n_seq, rows, attn_out);
}

int32_t launch_set_step(rmi_ctx* ctx, int* d_step, int value) {
  return rmi_run(ctx, "set_step", set_step_kernel, dim3(1), dim3(1), 0, d_step, value);
}
