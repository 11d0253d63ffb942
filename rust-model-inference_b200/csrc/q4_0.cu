// Q4_0 x Q8_0 matmul: exact int32 block dots of (nibble - 8) with the Q8_0 activation and the reference's
// f32 chain  sum += (f32(dot) * d) * scale  in block order.
//
// Reference (paths inside the reference project): src/ops/kernel/q4_0/scalar.rs:13-53; the AVX2 kernel
// (q4_0/avx2.rs:25-108) is bit-identical to it by contract (no FMA, block-by-block accumulation), so there is
// one semantics.  src/ops/kernel/q4_0/mod.rs:29-80 is the Kernel impl with its (ith, nth) partition.
//
// Device layout: the 18-byte blocks (f16 d | 16 nibble bytes), 2-byte aligned in a GGUF file, are padded to
// 20 bytes at upload (f16 d | 2 pad bytes | 16 nibble bytes) so that the nibble words are 4-byte aligned.
#include "common.cuh"
#include "kernels.cuh"

namespace {

constexpr int Q4_0_DEV_BYTES = 20;

// CTA = Q40_ROWS weight rows x MB activation rows, 32 blocks of K per step.  The order-free part runs in parallel: thread
// (row, block) forms the exact block dots of its weight block with every activation row and their scaled products; the
// ordered part, the sum over the blocks, is one thread per (row, activation row) out of shared memory.  A warp per row
// whose lane 0 fetched 32 products by shuffle spent about 900 cycles per step on that chain and read the weights once
// per activation row (24 rows of 3072 x 1024: 24 launches of 4.5 us; now one launch).  The weight blocks of the next
// step are requested before the products of the current one are summed.
constexpr int Q40_ROWS = 16, Q40_THREADS = 256, Q40_STEP = 32, Q40_PER = Q40_ROWS * Q40_STEP / Q40_THREADS;

template <int MB>
__host__ __device__ inline size_t q40_smem_bytes(size_t blocks) {
  // products [MB][rows][33] | activation pieces [MB][2][blocks] x 16 B | 8 * sum of the quants, scales [MB][blocks]
  return (size_t)MB * Q40_ROWS * (Q40_STEP + 1) * 4 + MB * blocks * (32 + 8) + 16;
}

template <int MB>
__global__ void __launch_bounds__(Q40_THREADS)
    q4_0_matmul_kernel(const uint8_t* __restrict__ w, size_t blocks, size_t n_rows, const uint8_t* __restrict__ xq,
                       const float* __restrict__ xs, float* __restrict__ out, size_t row_begin, size_t row_end) {
  extern __shared__ __align__(16) uint8_t q40_smem[];
  int4* x_s = reinterpret_cast<int4*>(q40_smem);                       // [MB][2][blocks]: bytes 0..15 / 16..31 of a block
  int* ys_s = reinterpret_cast<int*>(x_s + (size_t)MB * 2 * blocks);   // [MB][blocks]
  float* sc_s = reinterpret_cast<float*>(ys_s + (size_t)MB * blocks);  // [MB][blocks]
  float* prod = sc_s + (size_t)MB * blocks;                            // [MB][rows][Q40_STEP + 1]
  const int tid = threadIdx.x;
  const size_t row0 = row_begin + (size_t)blockIdx.x * Q40_ROWS, t0 = (size_t)blockIdx.y * MB;

  uint32_t q[Q40_PER][5];
  auto fetch = [&](size_t b0) {
#pragma unroll
    for (int k = 0; k < Q40_PER; k++) {
      const int item = tid + k * Q40_THREADS, r = item / Q40_STEP;
      const size_t b = b0 + item % Q40_STEP;
      const bool ok = row0 + r < row_end && b < blocks;
      const uint32_t* p = reinterpret_cast<const uint32_t*>(w + ((row0 + r) * blocks + b) * Q4_0_DEV_BYTES);
#pragma unroll
      for (int i = 0; i < 5; i++) q[k][i] = ok ? __ldg(p + i) : 0u;
    }
  };
  fetch(0);
  pdl_wait();  // the activations come from the preceding kernel
  for (size_t i = tid; i < (size_t)MB * blocks; i += Q40_THREADS) {
    const size_t m = i / blocks, b = i - m * blocks;
    const int4* src = reinterpret_cast<const int4*>(xq + ((t0 + m) * blocks + b) * 32);
    const int4 lo = __ldg(src), hi = __ldg(src + 1);
    x_s[(m * 2) * blocks + b] = lo;
    x_s[(m * 2 + 1) * blocks + b] = hi;
    int s = dp4a_s8(0x01010101, lo.x, dp4a_s8(0x01010101, lo.y, dp4a_s8(0x01010101, lo.z, dp4a_s8(0x01010101, lo.w, 0))));
    s = dp4a_s8(0x01010101, hi.x, dp4a_s8(0x01010101, hi.y, dp4a_s8(0x01010101, hi.z, dp4a_s8(0x01010101, hi.w, s))));
    ys_s[i] = -8 * s;  // sum (nibble - 8) * y = sum nibble * y - 8 * sum y
    sc_s[i] = __ldg(xs + (t0 + m) * blocks + b);
  }
  __syncthreads();
  float sum = 0.0f;
  const int sr = tid % Q40_ROWS, sm = tid / Q40_ROWS;  // the (row, activation row) this thread sums
  for (size_t b0 = 0; b0 < blocks; b0 += Q40_STEP) {
#pragma unroll
    for (int k = 0; k < Q40_PER; k++) {
      const int item = tid + k * Q40_THREADS, r = item / Q40_STEP, bl = item % Q40_STEP;
      const size_t b = b0 + bl;
      if (b < blocks) {
        const float d = f16_bits_to_f32((uint16_t)(q[k][0] & 0xffffu));
#pragma unroll
        for (int m = 0; m < MB; m++) {
          const int4 lo = x_s[(m * 2) * blocks + b], hi = x_s[(m * 2 + 1) * blocks + b];
          const int xl[4] = {lo.x, lo.y, lo.z, lo.w}, xh[4] = {hi.x, hi.y, hi.z, hi.w};
          int dot = ys_s[m * blocks + b];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            dot = dp4a_s8((int)(q[k][1 + i] & 0x0F0F0F0Fu), xl[i], dot);         // values 4i..4i+3: low nibbles
            dot = dp4a_s8((int)((q[k][1 + i] >> 4) & 0x0F0F0F0Fu), xh[i], dot);  // values 16+4i..: high nibbles
          }
          prod[(m * Q40_ROWS + r) * (Q40_STEP + 1) + bl] = __fmul_rn(__fmul_rn((float)dot, d), sc_s[m * blocks + b]);
        }
      }
    }
    if (b0 + Q40_STEP < blocks) fetch(b0 + Q40_STEP);
    __syncthreads();
    if (sm < MB) {
      const float* p = prod + (sm * Q40_ROWS + sr) * (Q40_STEP + 1);
      const int n = blocks - b0 < (size_t)Q40_STEP ? (int)(blocks - b0) : Q40_STEP;
      if (n == Q40_STEP) {
#pragma unroll
        for (int l = 0; l < Q40_STEP; l++) sum = __fadd_rn(sum, p[l]);
      } else {
        for (int l = 0; l < n; l++) sum = __fadd_rn(sum, p[l]);
      }
    }
    __syncthreads();
  }
  if (sm < MB && row0 + sr < row_end) out[(t0 + sm) * n_rows + row0 + sr] = sum;
}

// embedding_lookup_q4_0 (src/ops/embedding.rs:24-38): one CTA per requested row, ((nibble as f32) - 8) * d
__global__ void q4_0_embedding_kernel(const uint8_t* __restrict__ w, size_t blocks, const uint32_t* __restrict__ ids,
                                      float* __restrict__ out) {
  const uint8_t* row = w + (size_t)ids[blockIdx.x] * blocks * Q4_0_DEV_BYTES;
  for (size_t i = threadIdx.x; i < blocks * 16; i += blockDim.x) {
    const uint8_t* blk = row + (i / 16) * Q4_0_DEV_BYTES;
    const float d = f16_bits_to_f32(*reinterpret_cast<const uint16_t*>(blk));
    const uint8_t q = blk[4 + (i % 16)];
    float* o = out + (size_t)blockIdx.x * blocks * 32 + (i / 16) * 32 + (i % 16);
    o[0] = __fmul_rn(__fsub_rn((float)(q & 0x0F), 8.0f), d);
    o[16] = __fmul_rn(__fsub_rn((float)(q >> 4), 8.0f), d);
  }
}

}  // namespace

int32_t launch_q4_0_embedding(rmi_ctx* ctx, const rmi_weight* w, const uint32_t* ids, size_t m, float* out) {
  if (m == 0) return RMI_OK;
  q4_0_embedding_kernel<<<(unsigned)m, 256, 0, ctx->stream>>>(w->d_raw, w->n_in / 32, ids, out);
  return rmi_post_launch(ctx, "q4_0_embedding");
}

size_t q4_0_device_block_bytes() { return Q4_0_DEV_BYTES; }

template <int MB>
static int32_t q4_0_launch(rmi_ctx* ctx, const rmi_weight* w, const uint8_t* xq, const float* xs, size_t groups, float* out,
                           size_t row_begin, size_t row_end) {
  const size_t blocks = w->n_in / 32, smem = q40_smem_bytes<MB>(blocks);
  auto kern = q4_0_matmul_kernel<MB>;
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    rmi_set_error("cudaFuncSetAttribute(%zu B shared) failed", smem);
    return RMI_ERR_CUDA;
  }
  const dim3 grid((unsigned)((row_end - row_begin + Q40_ROWS - 1) / Q40_ROWS), (unsigned)groups);
  const cudaError_t le = rmi_launch(ctx, kern, grid, dim3(Q40_THREADS), smem, w->d_raw, blocks, w->n_rows, xq, xs, out,
                                          row_begin, row_end);
  if (le != cudaSuccess) {
    rmi_set_error("launch of q4_0_matmul failed: %s", cudaGetErrorString(le));
    return RMI_ERR_CUDA;
  }
  return rmi_post_launch(ctx, "q4_0_matmul");
}

int32_t launch_q4_0_matmul(rmi_ctx* ctx, const rmi_weight* w, const uint8_t* xq, const float* xs, size_t m, float* out,
                           size_t row_begin, size_t row_end) {
  if (row_begin >= row_end) return RMI_OK;
  const size_t blocks = w->n_in / 32, limit = ctx->smem_optin - 1024;
  RMI_REQUIRE(q40_smem_bytes<1>(blocks) <= limit, RMI_ERR_UNSUPPORTED, "n_in=%zu does not fit the Q4_0 activation buffer", w->n_in);
  size_t t = 0;
  while (t < m) {
    const size_t left = m - t;
    const bool eight = left >= 8 && q40_smem_bytes<8>(blocks) <= limit, four = left >= 4 && q40_smem_bytes<4>(blocks) <= limit;
    const size_t mb = eight ? 8 : (four ? 4 : 1), groups = left / mb;
    auto run = eight ? q4_0_launch<8> : (four ? q4_0_launch<4> : q4_0_launch<1>);
    RMI_TRY(run(ctx, w, xq + t * w->n_in, xs + t * blocks, groups, out + t * w->n_rows, row_begin, row_end));
    t += mb * groups;
  }
  return RMI_OK;
}
