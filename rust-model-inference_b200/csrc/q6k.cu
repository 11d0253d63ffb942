// Q6_K paths: the Q6_K x Q8_K row dot (exact integer sums, the reference's AVX2 or scalar f32 order), the
// Q8_0-activation path (dequantized row x dequantized activation) and the row dequantizer.
//
// Reference (paths inside the reference project):
//   src/ops/quant/mod.rs:530-569 (dequantize_row_q6_k), :640-692 and :964-1064 (vec_dot_q6k_q8k scalar / AVX2),
//   src/ops/kernel/q6_k.rs:22-80 (Kernel impl), :83-115 (matmul_q6_k_scalar_range).
//
// Device layout: the 210-byte super-blocks (ql[128] | qh[64] | i8 scales[16] | f16 d), which are only 2-byte
// aligned in a GGUF file, are padded to 224 bytes at upload so that every word load is aligned.
#include "common.cuh"
#include "kernels.cuh"

namespace {

constexpr int Q6K_DEV_BYTES = 224;

// four 6-bit values (0..63) as bytes of one word: positions 4L..4L+3 of vector (j, k) of a super-block
__device__ __forceinline__ uint32_t q6k_word(const uint8_t* blk, int j, int k, int L) {
  const uint32_t qlw = *reinterpret_cast<const uint32_t*>(blk + 64 * j + 32 * (k & 1) + 4 * L);
  const uint32_t qhw = *reinterpret_cast<const uint32_t*>(blk + 128 + 32 * j + 4 * L);
  return ((qlw >> (4 * (k >> 1))) & 0x0F0F0F0Fu) | (((qhw >> (2 * k)) & 0x03030303u) << 4);
}

// vec_dot_q6k_q8k in the scalar order for one weight row per warp, MP activation rows per pass.  Lane = (vq, L):
// L = lane % 8 selects bytes 4L..4L+3 of every 32-byte vector, vq = lane / 8 the vectors vq and vq + 4.
template <int MP>
__global__ void q6k_q8k_matmul_kernel(const uint8_t* __restrict__ w, size_t nb, size_t n_rows,
                                      const float* __restrict__ d8, const int8_t* __restrict__ q8,
                                      const int16_t* __restrict__ bs, float* __restrict__ out, size_t row_begin,
                                      size_t row_end) {
  const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  const size_t row = row_begin + warp;
  const size_t t0 = (size_t)blockIdx.y * MP;
  if (row >= row_end) return;
  const int L = lane & 7, vq = lane >> 3;
  const uint8_t* wrow = w + row * nb * Q6K_DEV_BYTES;
  float accs[MP][4];
#pragma unroll
  for (int m = 0; m < MP; m++)
#pragma unroll
    for (int k = 0; k < 4; k++) accs[m][k] = 0.0f;
  for (size_t i = 0; i < nb; i++) {
    const uint8_t* blk = wrow + i * Q6K_DEV_BYTES;
    const uint32_t qa = q6k_word(blk, 0, vq, L), qb = q6k_word(blk, 1, vq, L);   // vectors vq and vq + 4
    const int8_t* sc = reinterpret_cast<const int8_t*>(blk + 192);
    const int sca = sc[2 * vq + (L >= 4)], scb = sc[8 + 2 * vq + (L >= 4)];
    const float dw = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(blk + 208));
#pragma unroll
    for (int m = 0; m < MP; m++) {
      const size_t t = t0 + m;
      const int8_t* q8b = q8 + (t * nb + i) * 256;
      const int xa = *reinterpret_cast<const int*>(q8b + 32 * vq + 4 * L);
      const int xb = *reinterpret_cast<const int*>(q8b + 128 + 32 * vq + 4 * L);
      const float d = __fmul_rn(dw, d8[t * nb + i]);
      // mod.rs:675-687: aux32[e % 8] with e % 8 = 4 (L % 2) + byte
      int v[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int a6 = (int)((qa >> (8 * k)) & 0xff) - 32, b6 = (int)((qb >> (8 * k)) & 0xff) - 32;
        const int a8 = (int)(int8_t)((xa >> (8 * k)) & 0xff), b8 = (int)(int8_t)((xb >> (8 * k)) & 0xff);
        v[k] = sca * a8 * a6 + scb * b8 * b6;
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        v[k] += __shfl_xor_sync(0xffffffffu, v[k], 2);
        v[k] += __shfl_xor_sync(0xffffffffu, v[k], 4);
        v[k] += __shfl_xor_sync(0xffffffffu, v[k], 8);
        v[k] += __shfl_xor_sync(0xffffffffu, v[k], 16);
      }
#pragma unroll
      for (int k = 0; k < 4; k++) accs[m][k] = __fadd_rn(accs[m][k], __fmul_rn(d, (float)v[k]));
    }
  }
#pragma unroll
  for (int m = 0; m < MP; m++) {
    // sumf = sums[0] + ... + sums[7]: lane 0 holds sums[0..3], lane 1 sums[4..7]
    float hi[4];
#pragma unroll
    for (int k = 0; k < 4; k++) hi[k] = __shfl_sync(0xffffffffu, accs[m][k], 1);
    float r = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) r = __fadd_rn(r, accs[m][k]);
#pragma unroll
    for (int k = 0; k < 4; k++) r = __fadd_rn(r, hi[k]);
    if (lane == 0) out[(t0 + m) * n_rows + row] = r;
  }
}

// The AVX2 order for MB activation rows with the weight rows streamed through shared memory.  The row kernel above walks
// a row with one dependent load after another and reached 2.1 TB/s on a 151936 x 1024 head (63 us); what bounds this
// path is reading the weights, so every warp owns four consecutive rows and a private ring of bulk copies (a stage is
// up to Q6S_SB super-blocks of each row), which keeps Q6S_S * 3.5 KiB per warp in flight whatever the row length.
// Lane = (quad q = row, AVX2 lane L): lane L's integer sum over the eight 32-byte vectors of a super-block needs no
// shuffle.  The activation rows are staged once per CTA, permuted so that a lane finds its eight words of a super-block
// in two 16-byte pieces; the stage's rows start eight banks apart.
constexpr int Q6S_WARPS = 4, Q6S_TN = 4 * Q6S_WARPS, Q6S_SB = 4, Q6S_S = 4;
constexpr int Q6S_ROW_BYTES = Q6S_SB * Q6K_DEV_BYTES + 32, Q6S_STAGE_BYTES = 4 * Q6S_ROW_BYTES;
constexpr int Q6S_RING_BYTES = Q6S_WARPS * Q6S_S * Q6S_STAGE_BYTES;
__host__ __device__ inline size_t q6s_smem_bytes(size_t mb, size_t nb) {
  return (size_t)Q6S_RING_BYTES + 128 + mb * nb * (256 + 64 + 4);
}

template <int MB>
__global__ void __launch_bounds__(32 * Q6S_WARPS)
    q6k_q8k_stream_kernel(const uint8_t* __restrict__ w, size_t nb, size_t n_rows, const float* __restrict__ d8,
                          const int8_t* __restrict__ q8, const int16_t* __restrict__ bs, float* __restrict__ out,
                          size_t row_begin, size_t row_end, size_t n_tiles, rmi_dev_status* status) {
  extern __shared__ __align__(128) uint8_t q6s_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int L = lane & 7, q = lane >> 3;
  uint8_t* ring = q6s_smem + warp * (Q6S_S * Q6S_STAGE_BYTES);
  uint64_t* bar = reinterpret_cast<uint64_t*>(q6s_smem + Q6S_RING_BYTES) + warp * Q6S_S;
  int* xq_s = reinterpret_cast<int*>(q6s_smem + Q6S_RING_BYTES + 128);   // [MB][nb][2][8 lanes][4] words
  int2* xb_s = reinterpret_cast<int2*>(xq_s + (size_t)MB * nb * 64);     // [MB][nb][8 lanes]: bsums 2 L and 2 L + 1
  float* xd_s = reinterpret_cast<float*>(xb_s + (size_t)MB * nb * 8);    // [MB][nb]
  const uint32_t bar_a = (uint32_t)__cvta_generic_to_shared(bar), ring_a = (uint32_t)__cvta_generic_to_shared(ring);
  const int n_chunks = (int)((nb + Q6S_SB - 1) / Q6S_SB);
  const size_t my_tiles = blockIdx.x < n_tiles ? (n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const size_t n_items = my_tiles * (size_t)n_chunks;
  const size_t t0 = (size_t)blockIdx.y * MB;

  size_t tile_i = blockIdx.x;   // tile and chunk of the next item to request
  int chunk_i = 0;
  auto issue = [&](size_t j) {
    const size_t i0 = (size_t)chunk_i * Q6S_SB;
    const uint32_t n = (uint32_t)(nb - i0 < (size_t)Q6S_SB ? nb - i0 : (size_t)Q6S_SB);
    const uint32_t st = (uint32_t)(j % Q6S_S), bytes = n * Q6K_DEV_BYTES;
    if (lane == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_a + 8 * st), "r"(bytes * 4u) : "memory");
    __syncwarp();
    if (lane < 4) {
      size_t row = row_begin + tile_i * Q6S_TN + warp * 4 + lane;
      if (row >= row_end) row = row_end - 1;   // rows past the range repeat the last one (never stored)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       ring_a + st * (uint32_t)Q6S_STAGE_BYTES + (uint32_t)lane * Q6S_ROW_BYTES),
                   "l"(w + (row * nb + i0) * Q6K_DEV_BYTES), "r"(bytes), "r"(bar_a + 8 * st)
                   : "memory");
    }
    if (++chunk_i == n_chunks) {
      chunk_i = 0;
      tile_i += gridDim.x;
    }
  };
  if (lane == 0) {
    for (int i = 0; i < Q6S_S; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a + 8 * i));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  for (size_t j = 0; j < n_items && j < (size_t)Q6S_S; j++) issue(j);
  pdl_wait();  // the weights above are never written; the activations come from the preceding kernel
  {
    // word 32 j + 8 k + l of a super-block (half j, vector k of the half, lane l) goes to 32 j + 4 l + k
    const int* src = reinterpret_cast<const int*>(q8 + t0 * nb * 256);
    for (size_t idx = tid; idx < (size_t)MB * nb * 64; idx += 32 * Q6S_WARPS) {
      const int ws = (int)(idx & 63), k = (ws >> 3) & 3, l = ws & 7;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(
                       xq_s + (idx & ~(size_t)63) + (ws & 32) + 4 * l + k)),
                   "l"(src + idx)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (size_t idx = tid; idx < (size_t)MB * nb * 8; idx += 32 * Q6S_WARPS) {
      const uint32_t b2 = __ldg(reinterpret_cast<const uint32_t*>(bs + t0 * nb * 16) + idx);
      xb_s[idx] = make_int2((int)(int16_t)(b2 & 0xffff), (int)(int16_t)(b2 >> 16));
    }
    for (size_t idx = tid; idx < (size_t)MB * nb; idx += 32 * Q6S_WARPS) xd_s[idx] = __ldg(d8 + t0 * nb + idx);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();

  const uint64_t limit_ns = status->limit_ns;
  const int hi = L >= 4;
  float acc[MB];
  size_t tile = blockIdx.x;
  int c = 0;
  for (size_t j = 0; j < n_items; j++) {
    const uint32_t st = (uint32_t)(j % Q6S_S), parity = (uint32_t)((j / Q6S_S) & 1);
    if (c == 0) {
#pragma unroll
      for (int b = 0; b < MB; b++) acc[b] = 0.0f;
    }
    if (!mbar_wait_limited(bar_a + 8 * st, parity, limit_ns)) {
      // the copies in flight target this CTA's own shared memory and are dropped with it
      if (atomicCAS(&status->code, 0, RMI_ERR_TIMEOUT) == 0) {
        status->where = 14;
        status->detail = (int)j;
      }
      return;
    }
    const size_t i0 = (size_t)c * Q6S_SB;
    const int n = (int)(nb - i0 < (size_t)Q6S_SB ? nb - i0 : (size_t)Q6S_SB);
    const uint8_t* row_s = ring + (size_t)st * Q6S_STAGE_BYTES + (size_t)q * Q6S_ROW_BYTES;
#pragma unroll
    for (int u = 0; u < Q6S_SB; u++) {
      if (u >= n) break;  // uniform
      const size_t i = i0 + u;
      const uint8_t* blk = row_s + u * Q6K_DEV_BYTES;
      const uint4 scw = *reinterpret_cast<const uint4*>(blk + 192);   // the 16 signed scales
      const uint32_t sw[4] = {scw.x, scw.y, scw.z, scw.w};
      const float dw = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(blk + 208));
      int qv[8], sc[8];
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const uint32_t q0 = *reinterpret_cast<const uint32_t*>(blk + 64 * half + 4 * L);
        const uint32_t q1 = *reinterpret_cast<const uint32_t*>(blk + 64 * half + 32 + 4 * L);
        const uint32_t qh = *reinterpret_cast<const uint32_t*>(blk + 128 + 32 * half + 4 * L);
        qv[4 * half + 0] = (int)((q0 & 0x0F0F0F0Fu) | ((qh << 4) & 0x30303030u));
        qv[4 * half + 1] = (int)((q1 & 0x0F0F0F0Fu) | ((qh << 2) & 0x30303030u));
        qv[4 * half + 2] = (int)(((q0 >> 4) & 0x0F0F0F0Fu) | (qh & 0x30303030u));
        qv[4 * half + 3] = (int)(((q1 >> 4) & 0x0F0F0F0Fu) | ((qh >> 2) & 0x30303030u));
      }
#pragma unroll
      for (int k = 0; k < 8; k++) sc[k] = (int)(int8_t)(sw[k >> 1] >> (16 * (k & 1) + 8 * hi));
      const uint32_t swl = L < 4 ? (L < 2 ? sw[0] : sw[1]) : (L < 6 ? sw[2] : sw[3]);   // scales 2 L and 2 L + 1
      const int sub_a = (int)(int8_t)(swl >> (16 * (L & 1))), sub_b = (int)(int8_t)(swl >> (16 * (L & 1) + 8));
#pragma unroll
      for (int b = 0; b < MB; b++) {
        const size_t rb = (size_t)b * nb + i;
        const int4 xa = *reinterpret_cast<const int4*>(xq_s + rb * 64 + 4 * L);
        const int4 xb = *reinterpret_cast<const int4*>(xq_s + rb * 64 + 32 + 4 * L);
        const int2 ss = xb_s[rb * 8 + L];
        int v = sc[0] * dp4a_s8(qv[0], xa.x, 0) + sc[1] * dp4a_s8(qv[1], xa.y, 0);   // mod.rs:998-1062
        v += sc[2] * dp4a_s8(qv[2], xa.z, 0) + sc[3] * dp4a_s8(qv[3], xa.w, 0);
        v += sc[4] * dp4a_s8(qv[4], xb.x, 0) + sc[5] * dp4a_s8(qv[5], xb.y, 0);
        v += sc[6] * dp4a_s8(qv[6], xb.z, 0) + sc[7] * dp4a_s8(qv[7], xb.w, 0);
        v -= 32 * (ss.x * sub_a + ss.y * sub_b);
        acc[b] = __fmaf_rn(__fmul_rn(dw, xd_s[rb]), (float)v, acc[b]);
      }
    }
    __syncwarp();  // every lane is done with the stage
    if (j + Q6S_S < n_items) issue(j + Q6S_S);
    if (c == n_chunks - 1) {
      const size_t row = row_begin + tile * Q6S_TN + warp * 4 + q;
#pragma unroll
      for (int b = 0; b < MB; b++) {
        // hsum_ps over the eight lanes (dot.rs:447-456)
        const float s = __fadd_rn(__shfl_xor_sync(0xffffffffu, acc[b], 4), acc[b]);
        const float uu = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 1));
        const float r = __fadd_rn(uu, __shfl_xor_sync(0xffffffffu, uu, 2));
        if (L == 0 && row < row_end) out[(t0 + b) * n_rows + row] = r;
      }
    }
    if (++c == n_chunks) {
      c = 0;
      tile += gridDim.x;
    }
  }
}

// matmul_q6_k_scalar_range: dequantized row (d*sc)*q times the dequantized Q8_0 activation q8*scale, summed by a
// warp tree (the reference sums sequentially in f32; tolerance 1e-4).  One warp per weight row.
__global__ void q6k_prequant_matmul_kernel(const uint8_t* __restrict__ w, size_t nb, size_t n_rows,
                                           const uint8_t* __restrict__ xq, const float* __restrict__ xs,
                                           float* __restrict__ out, size_t row_begin, size_t row_end) {
  const size_t row = row_begin + ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  const size_t t = blockIdx.y;
  if (row >= row_end) return;
  const int L = lane & 7, vq = lane >> 3;
  const size_t K = nb * 256;
  const uint8_t* wrow = w + row * nb * Q6K_DEV_BYTES;
  float acc = 0.0f;
  for (size_t i = 0; i < nb; i++) {
    const uint8_t* blk = wrow + i * Q6K_DEV_BYTES;
    const int8_t* sc = reinterpret_cast<const int8_t*>(blk + 192);
    const float dw = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(blk + 208));
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const uint32_t q = q6k_word(blk, j, vq, L);
      const int e0 = 128 * j + 32 * vq + 4 * L;
      const float ds = __fmul_rn(dw, (float)sc[e0 / 16]);
      const int xw = *reinterpret_cast<const int*>(xq + t * K + i * 256 + e0);
      const float xsc = xs[t * (K / 32) + (i * 256 + e0) / 32];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float wv = __fmul_rn(ds, (float)((int)((q >> (8 * k)) & 0xff) - 32));
        const float xv = __fmul_rn((float)(int)(int8_t)((xw >> (8 * k)) & 0xff), xsc);
        acc = __fmaf_rn(wv, xv, acc);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) out[t * n_rows + row] = acc;
}

__global__ void q6k_dequantize_kernel(const uint8_t* __restrict__ w, size_t n_superblocks, float* __restrict__ out) {
  const size_t sb = (size_t)blockIdx.x;
  if (sb >= n_superblocks) return;
  const uint8_t* blk = w + sb * Q6K_DEV_BYTES;
  const int e = threadIdx.x;  // 256 threads: one value each
  const int j = e / 128, r = e % 128, k = r / 32, l = r % 32;
  const uint8_t qlb = blk[64 * j + 32 * (k & 1) + l], qhb = blk[128 + 32 * j + l];
  const int q = (int)(((qlb >> (4 * (k >> 1))) & 0xF) | (((qhb >> (2 * k)) & 3) << 4)) - 32;
  const float d = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(blk + 208));
  const float sc = (float)(int)(int8_t)blk[192 + e / 16];
  out[sb * 256 + e] = __fmul_rn(__fmul_rn(d, sc), (float)q);
}

// embedding_lookup_q6_k (src/ops/embedding.rs:40-47): dequantize_row_q6_k of the requested rows;
// grid (super-blocks per row, rows), 256 threads = one value each
__global__ void q6k_embedding_kernel(const uint8_t* __restrict__ w, size_t nb, const uint32_t* __restrict__ ids,
                                     float* __restrict__ out) {
  const uint8_t* blk = w + ((size_t)ids[blockIdx.y] * nb + blockIdx.x) * Q6K_DEV_BYTES;
  const int e = threadIdx.x;
  const int j = e / 128, r = e % 128, k = r / 32, l = r % 32;
  const uint8_t qlb = blk[64 * j + 32 * (k & 1) + l], qhb = blk[128 + 32 * j + l];
  const int q = (int)(((qlb >> (4 * (k >> 1))) & 0xF) | (((qhb >> (2 * k)) & 3) << 4)) - 32;
  const float d = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(blk + 208));
  const float sc = (float)(int)(int8_t)blk[192 + e / 16];
  out[((size_t)blockIdx.y * nb + blockIdx.x) * 256 + e] = __fmul_rn(__fmul_rn(d, sc), (float)q);
}

template <int MP>
void q6k_q8k_launch(rmi_ctx* ctx, const rmi_weight* w, const float* d8, const int8_t* qs, const int16_t* bsums,
                    size_t groups, float* out, size_t row_begin, size_t row_end) {
  const size_t rows = row_end - row_begin, nb = w->n_in / 256;
  dim3 grid((unsigned)((rows + 3) / 4), (unsigned)groups);
  q6k_q8k_matmul_kernel<MP><<<grid, 128, 0, ctx->stream>>>(w->d_raw, nb, w->n_rows, d8, qs, bsums, out, row_begin, row_end);
}

template <int MB>
int32_t q6k_stream_launch(rmi_ctx* ctx, const rmi_weight* w, const float* d8, const int8_t* qs, const int16_t* bsums,
                          size_t groups, float* out, size_t row_begin, size_t row_end) {
  const size_t nb = w->n_in / 256, smem = q6s_smem_bytes(MB, nb);
  const size_t n_tiles = (row_end - row_begin + Q6S_TN - 1) / Q6S_TN;
  auto kern = q6k_q8k_stream_kernel<MB>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    rmi_set_error("cudaFuncSetAttribute(%zu B shared) failed", smem);
    return RMI_ERR_CUDA;
  }
  size_t per_sm = (ctx->smem_optin + 1024) / (smem + 1024);
  if (per_sm < 1) per_sm = 1;
  size_t grid = (size_t)ctx->sm_count * per_sm;
  if (grid > n_tiles) grid = n_tiles;
  const size_t tiles_per_cta = (n_tiles + grid - 1) / grid;
  grid = (n_tiles + tiles_per_cta - 1) / tiles_per_cta;   // every CTA walks the same number of tiles
  const cudaError_t le = rmi_launch(ctx, kern, dim3((unsigned)grid, (unsigned)groups), dim3(32 * Q6S_WARPS), smem, w->d_raw,
                                          nb, w->n_rows, d8, qs, bsums, out, row_begin, row_end, n_tiles, ctx->d_status);
  if (le != cudaSuccess) {
    rmi_set_error("launch of q6k_q8k_stream failed: %s", cudaGetErrorString(le));
    return RMI_ERR_CUDA;
  }
  return rmi_post_launch(ctx, "q6k_q8k_stream");
}

}  // namespace

size_t q6k_device_block_bytes() { return Q6K_DEV_BYTES; }

int32_t launch_q6k_embedding(rmi_ctx* ctx, const rmi_weight* w, const uint32_t* ids, size_t m, float* out) {
  if (m == 0) return RMI_OK;
  q6k_embedding_kernel<<<dim3((unsigned)(w->n_in / 256), (unsigned)m), 256, 0, ctx->stream>>>(w->d_raw, w->n_in / 256, ids, out);
  return rmi_post_launch(ctx, "q6k_embedding");
}

int32_t launch_q6k_q8k_matmul(rmi_ctx* ctx, const rmi_weight* w, const float* d8, const int8_t* qs,
                              const int16_t* bsums, size_t m, float* out, size_t row_begin, size_t row_end) {
  if (m == 0 || row_begin >= row_end) return RMI_OK;
  const size_t nb = w->n_in / 256;
  size_t t = 0;
  if (ctx->sem != RMI_SEM_SCALAR) {
    while (t < m) {
      const size_t left = m - t;
      size_t mb = left >= 8 ? 8 : (left >= 4 ? 4 : (left >= 2 ? 2 : 1));
      while (mb > 1 && q6s_smem_bytes(mb, nb) > ctx->smem_optin - 1024) mb >>= 1;
      RMI_REQUIRE(q6s_smem_bytes(mb, nb) <= ctx->smem_optin - 1024, RMI_ERR_UNSUPPORTED,
                  "n_in=%zu does not fit the Q6_K x Q8_K shared-memory buffers", w->n_in);
      auto run = mb == 8 ? q6k_stream_launch<8> : (mb == 4 ? q6k_stream_launch<4> : (mb == 2 ? q6k_stream_launch<2> : q6k_stream_launch<1>));
      const size_t groups = left / mb;
      RMI_TRY(run(ctx, w, d8 + t * nb, qs + t * nb * 256, bsums + t * nb * 16, groups, out + t * w->n_rows, row_begin, row_end));
      t += mb * groups;
    }
    return RMI_OK;
  }
  if (m >= 4) {
    q6k_q8k_launch<4>(ctx, w, d8, qs, bsums, m / 4, out, row_begin, row_end);
    RMI_TRY(rmi_post_launch(ctx, "q6k_q8k_matmul"));
    t = m / 4 * 4;
  }
  if (t < m) {
    q6k_q8k_launch<1>(ctx, w, d8 + t * nb, qs + t * nb * 256, bsums + t * nb * 16, m - t, out + t * w->n_rows, row_begin, row_end);
    RMI_TRY(rmi_post_launch(ctx, "q6k_q8k_matmul"));
  }
  return RMI_OK;
}

int32_t launch_q6k_prequant_matmul(rmi_ctx* ctx, const rmi_weight* w, const uint8_t* xq, const float* xs, size_t m,
                                   float* out, size_t row_begin, size_t row_end) {
  if (m == 0 || row_begin >= row_end) return RMI_OK;
  dim3 grid((unsigned)((row_end - row_begin + 3) / 4), (unsigned)m);
  q6k_prequant_matmul_kernel<<<grid, 128, 0, ctx->stream>>>(w->d_raw, w->n_in / 256, w->n_rows, xq, xs, out, row_begin, row_end);
  return rmi_post_launch(ctx, "q6k_prequant_matmul");
}

int32_t launch_q6k_dequantize(rmi_ctx* ctx, const rmi_weight* w, float* out) {
  const size_t nsb = w->n_rows * (w->n_in / 256);
  if (nsb == 0) return RMI_OK;
  q6k_dequantize_kernel<<<(unsigned)nsb, 256, 0, ctx->stream>>>(w->d_raw, nsb, out);
  return rmi_post_launch(ctx, "q6k_dequantize");
}
