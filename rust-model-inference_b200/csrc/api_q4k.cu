// Host- and device-pointer entry points of the Q4_K paths.
#include "common.cuh"
#include "kernels.cuh"

extern "C" int32_t rmi_quantize_q8_k(rmi_ctx* ctx, const float* x, size_t m, size_t n, float* d, int8_t* qs,
                                     int16_t* bsums) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_REQUIRE(n % 256 == 0, RMI_ERR_BAD_SHAPE, "n=%zu is not a multiple of 256", n);
  if (m * n == 0) return RMI_OK;
  RMI_REQUIRE(x && d && qs && bsums, RMI_ERR_BAD_HANDLE, "rmi_quantize_q8_k: null buffer");
  RMI_REQUIRE(ctx->sem != RMI_SEM_NEON, RMI_ERR_UNSUPPORTED, "the reference has no NEON Q8_K quantizer; use AVX2 or SCALAR");
  std::lock_guard<std::mutex> lock(ctx->mu);
  const size_t nb = m * n / 256;
  float *dx, *dd;
  int8_t* dq;
  int16_t* db;
  RMI_TRY(rmi_scratch(ctx, 5, m * n * 4, (void**)&dx));
  RMI_TRY(rmi_scratch(ctx, 0, m * n, (void**)&dq));
  RMI_TRY(rmi_scratch(ctx, 1, nb * 4, (void**)&dd));
  RMI_TRY(rmi_scratch(ctx, 4, nb * 32, (void**)&db));
  RMI_CUDA_CHECK(cudaMemcpyAsync(dx, x, m * n * 4, cudaMemcpyHostToDevice, ctx->stream));
  RMI_TRY(launch_q8k_quantize(ctx, dx, m, n, dd, dq, db));
  RMI_CUDA_CHECK(cudaMemcpyAsync(d, dd, nb * 4, cudaMemcpyDeviceToHost, ctx->stream));
  RMI_CUDA_CHECK(cudaMemcpyAsync(qs, dq, m * n, cudaMemcpyDeviceToHost, ctx->stream));
  RMI_CUDA_CHECK(cudaMemcpyAsync(bsums, db, nb * 32, cudaMemcpyDeviceToHost, ctx->stream));
  RMI_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
  return RMI_OK;
}

// Quantize to Q8_K, then Q4_K x Q8_K; caller holds ctx->mu.  The tensor-core kernel exists for the AVX2 order only; up to 16
// rows cost it what one does, so it takes over from the passes of the streaming kernels at three (4096 x 4096: 1, 2, 4, 8
// rows streamed 10, 10, 16, 20 us; on the tensor cores 10).
static constexpr size_t Q4K_Q8K_MMA_MIN_M = 3;

static int32_t q4k_q8k_device(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, float* out, size_t row_begin, size_t row_end) {
  if (m >= Q4K_Q8K_MMA_MIN_M && ctx->sem == RMI_SEM_AVX2 && q4k_mma_prepare(ctx, w, false)) {
    uint8_t* xrec;
    RMI_TRY(rmi_scratch(ctx, 0, q4k_mma_x_bytes(w, m, false), (void**)&xrec));
    return launch_q4k_q8k_mma(ctx, w, x, m, xrec, out, row_begin, row_end);
  }
  const size_t n = w->n_in, nb = m * n / 256;
  float* dd;
  int8_t* dq;
  int16_t* db;
  RMI_TRY(rmi_scratch(ctx, 0, m * n, (void**)&dq));
  RMI_TRY(rmi_scratch(ctx, 1, nb * 4, (void**)&dd));
  RMI_TRY(rmi_scratch(ctx, 4, nb * 32, (void**)&db));
  RMI_TRY(launch_q8k_quantize(ctx, x, m, n, dd, dq, db));
  return launch_q4k_q8k_matmul(ctx, w, dd, dq, db, m, out, row_begin, row_end);
}

extern "C" int32_t rmi_matmul_q4_k_q8k(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, float* output,
                                       size_t row_begin, size_t row_end) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q4_K));
  RMI_REQUIRE(row_begin <= row_end && row_end <= w->n_rows, RMI_ERR_BAD_SHAPE, "row range [%zu,%zu) outside [0,%zu)",
              row_begin, row_end, w->n_rows);
  if (m == 0 || row_begin == row_end) return RMI_OK;
  RMI_REQUIRE(x && output, RMI_ERR_BAD_HANDLE, "rmi_matmul_q4_k_q8k: null buffer");
  RMI_REQUIRE(ctx->sem != RMI_SEM_NEON, RMI_ERR_UNSUPPORTED, "the reference has no NEON Q4_K x Q8_K kernel; use AVX2 or SCALAR");
  std::lock_guard<std::mutex> lock(ctx->mu);
  const size_t n = w->n_in, nr = row_end - row_begin;
  float *dx, *dout;
  RMI_TRY(host_in(ctx, x, m * n * 4, 5, true, (void**)&dx));
  RMI_TRY(rmi_scratch(ctx, 6, m * w->n_rows * 4, (void**)&dout));
  RMI_TRY(q4k_q8k_device(ctx, w, dx, m, dout, row_begin, row_end));
  return host_out(ctx, output + row_begin, dout + row_begin, m, nr * 4, w->n_rows * 4);
}

extern "C" int32_t rmi_matmul_q4_k_q8k_dev(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, float* output) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q4_K));
  if (m == 0 || w->n_rows == 0) return RMI_OK;
  RMI_REQUIRE(x && output, RMI_ERR_BAD_HANDLE, "rmi_matmul_q4_k_q8k_dev: null buffer");
  RMI_REQUIRE(ctx->sem != RMI_SEM_NEON, RMI_ERR_UNSUPPORTED, "the reference has no NEON Q4_K x Q8_K kernel; use AVX2 or SCALAR");
  std::lock_guard<std::mutex> lock(ctx->mu);
  return q4k_q8k_device(ctx, w, x, m, output, 0, w->n_rows);
}

// The time of the tensor-core kernel for few rows is that of one CTA walking K, whatever the number of weight rows that the
// SMs hold at once: 23 us for K = 4096 with 4096 or 11008 rows, where 8 activation rows take the streaming kernel 18 and
// 47 us, 12 take it 33 and 73.
static bool q4k_dequant_on_mma(const rmi_weight* w, size_t m) { return m >= 9 || (m >= 5 && w->n_rows >= 8192); }

static int32_t q4k_dequant_device(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, float* out) {
  if (!q4k_dequant_on_mma(w, m) || !q4k_mma_prepare(ctx, w, true)) return launch_q4k_dequant_matmul(ctx, w, x, m, out);
  uint8_t* xrec;
  RMI_TRY(rmi_scratch(ctx, 0, q4k_mma_x_bytes(w, m, true), (void**)&xrec));
  return launch_q4k_dequant_mma(ctx, w, x, m, xrec, out);
}

extern "C" int32_t rmi_matmul_q4_k_dequant_dev(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m,
                                               float* output) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q4_K));
  RMI_REQUIRE(((uintptr_t)x & 15) == 0, RMI_ERR_BAD_SHAPE, "device input must be 16-byte aligned");
  std::lock_guard<std::mutex> lock(ctx->mu);
  return q4k_dequant_device(ctx, w, x, m, output);
}

extern "C" int32_t rmi_matmul_q4_k_dequant(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, float* output) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q4_K));
  if (m == 0 || w->n_rows == 0) return RMI_OK;
  RMI_REQUIRE(x && output, RMI_ERR_BAD_HANDLE, "rmi_matmul_q4_k_dequant: null buffer");
  std::lock_guard<std::mutex> lock(ctx->mu);
  float *dx, *dout;
  RMI_TRY(host_in(ctx, x, m * w->n_in * 4, 5, false, (void**)&dx));
  RMI_TRY(rmi_scratch(ctx, 6, m * w->n_rows * 4, (void**)&dout));
  RMI_TRY(q4k_dequant_device(ctx, w, dx, m, dout));
  return host_out(ctx, output, dout, 1, m * w->n_rows * 4, 0);
}

extern "C" int32_t rmi_dequantize_q4_k(rmi_ctx* ctx, const rmi_weight* w, float* output) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q4_K));
  if (w->n_rows == 0) return RMI_OK;
  RMI_REQUIRE(output != nullptr, RMI_ERR_BAD_HANDLE, "rmi_dequantize_q4_k: null buffer");
  std::lock_guard<std::mutex> lock(ctx->mu);
  float* dout;
  RMI_TRY(rmi_scratch(ctx, 6, w->n_rows * w->n_in * 4, (void**)&dout));
  RMI_TRY(launch_q4k_dequantize(ctx, w, dout));
  RMI_CUDA_CHECK(cudaMemcpyAsync(output, dout, w->n_rows * w->n_in * 4, cudaMemcpyDeviceToHost, ctx->stream));
  RMI_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
  return RMI_OK;
}

// ---------------------------------------------------------------- Q6_K

extern "C" int32_t rmi_matmul_q6_k_q8k(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, float* output,
                                       size_t row_begin, size_t row_end) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q6_K));
  RMI_REQUIRE(row_begin <= row_end && row_end <= w->n_rows, RMI_ERR_BAD_SHAPE, "row range [%zu,%zu) outside [0,%zu)",
              row_begin, row_end, w->n_rows);
  if (m == 0 || row_begin == row_end) return RMI_OK;
  RMI_REQUIRE(x && output, RMI_ERR_BAD_HANDLE, "rmi_matmul_q6_k_q8k: null buffer");
  RMI_REQUIRE(ctx->sem != RMI_SEM_NEON, RMI_ERR_UNSUPPORTED, "the reference has no NEON Q6_K x Q8_K kernel; use AVX2 or SCALAR");
  std::lock_guard<std::mutex> lock(ctx->mu);
  const size_t n = w->n_in, nb = m * n / 256, nr = row_end - row_begin;
  float *dx, *dd, *dout;
  int8_t* dq;
  int16_t* db;
  RMI_TRY(host_in(ctx, x, m * n * 4, 5, true, (void**)&dx));
  RMI_TRY(rmi_scratch(ctx, 0, m * n, (void**)&dq));
  RMI_TRY(rmi_scratch(ctx, 1, nb * 4, (void**)&dd));
  RMI_TRY(rmi_scratch(ctx, 4, nb * 32, (void**)&db));
  RMI_TRY(rmi_scratch(ctx, 6, m * w->n_rows * 4, (void**)&dout));
  RMI_TRY(launch_q8k_quantize(ctx, dx, m, n, dd, dq, db));
  RMI_TRY(launch_q6k_q8k_matmul(ctx, w, dd, dq, db, m, dout, row_begin, row_end));
  return host_out(ctx, output + row_begin, dout + row_begin, m, nr * 4, w->n_rows * 4);
}

extern "C" int32_t rmi_matmul_q6_k_prequantized(rmi_ctx* ctx, const rmi_weight* w, const uint8_t* q8, const float* scales,
                                                size_t m, float* output, size_t row_begin, size_t row_end) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q6_K));
  RMI_REQUIRE(row_begin <= row_end && row_end <= w->n_rows, RMI_ERR_BAD_SHAPE, "row range [%zu,%zu) outside [0,%zu)",
              row_begin, row_end, w->n_rows);
  if (m == 0 || row_begin == row_end) return RMI_OK;
  RMI_REQUIRE(q8 && scales && output, RMI_ERR_BAD_HANDLE, "rmi_matmul_q6_k_prequantized: null buffer");
  std::lock_guard<std::mutex> lock(ctx->mu);
  const size_t n = w->n_in, nr = row_end - row_begin;
  uint8_t* dq;
  float *ds, *dout;
  RMI_TRY(host_in(ctx, q8, m * n, 0, false, (void**)&dq));
  RMI_TRY(rmi_scratch(ctx, 1, m * (n / 32) * 4, (void**)&ds));
  RMI_TRY(rmi_scratch(ctx, 6, m * w->n_rows * 4, (void**)&dout));
  RMI_CUDA_CHECK(cudaMemcpyAsync(ds, scales, m * (n / 32) * 4, cudaMemcpyHostToDevice, ctx->stream));
  RMI_TRY(launch_q6k_prequant_matmul(ctx, w, dq, ds, m, dout, row_begin, row_end));
  return host_out(ctx, output + row_begin, dout + row_begin, m, nr * 4, w->n_rows * 4);
}

extern "C" int32_t rmi_dequantize_q6_k(rmi_ctx* ctx, const rmi_weight* w, float* output) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q6_K));
  if (w->n_rows == 0) return RMI_OK;
  RMI_REQUIRE(output != nullptr, RMI_ERR_BAD_HANDLE, "rmi_dequantize_q6_k: null buffer");
  std::lock_guard<std::mutex> lock(ctx->mu);
  float* dout;
  RMI_TRY(rmi_scratch(ctx, 6, w->n_rows * w->n_in * 4, (void**)&dout));
  RMI_TRY(launch_q6k_dequantize(ctx, w, dout));
  RMI_CUDA_CHECK(cudaMemcpyAsync(output, dout, w->n_rows * w->n_in * 4, cudaMemcpyDeviceToHost, ctx->stream));
  RMI_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
  return RMI_OK;
}

// ---------------------------------------------------------------- Q4_0

extern "C" int32_t rmi_matmul_q4_0_prequantized(rmi_ctx* ctx, const rmi_weight* w, const uint8_t* q8, const float* scales,
                                                size_t m, float* output, size_t row_begin, size_t row_end) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q4_0));
  RMI_REQUIRE(row_begin <= row_end && row_end <= w->n_rows, RMI_ERR_BAD_SHAPE, "row range [%zu,%zu) outside [0,%zu)",
              row_begin, row_end, w->n_rows);
  if (m == 0 || row_begin == row_end) return RMI_OK;
  RMI_REQUIRE(q8 && scales && output, RMI_ERR_BAD_HANDLE, "rmi_matmul_q4_0_prequantized: null buffer");
  std::lock_guard<std::mutex> lock(ctx->mu);
  const size_t n = w->n_in, nr = row_end - row_begin;
  uint8_t* dq;
  float *ds, *dout;
  RMI_TRY(host_in(ctx, q8, m * n, 0, false, (void**)&dq));
  RMI_TRY(rmi_scratch(ctx, 1, m * (n / 32) * 4, (void**)&ds));
  RMI_TRY(rmi_scratch(ctx, 6, m * w->n_rows * 4, (void**)&dout));
  RMI_CUDA_CHECK(cudaMemcpyAsync(ds, scales, m * (n / 32) * 4, cudaMemcpyHostToDevice, ctx->stream));
  RMI_TRY(launch_q4_0_matmul(ctx, w, dq, ds, m, dout, row_begin, row_end));
  return host_out(ctx, output + row_begin, dout + row_begin, m, nr * 4, w->n_rows * 4);
}

extern "C" int32_t rmi_matmul_q4_0(rmi_ctx* ctx, const rmi_weight* w, const float* x, size_t m, float* output) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, RMI_GGML_Q4_0));
  if (m == 0 || w->n_rows == 0) return RMI_OK;
  RMI_REQUIRE(x && output, RMI_ERR_BAD_HANDLE, "rmi_matmul_q4_0: null buffer");
  std::lock_guard<std::mutex> lock(ctx->mu);
  const size_t n = w->n_in;
  uint8_t* dq;
  float *dx, *ds, *dout;
  RMI_TRY(host_in(ctx, x, m * n * 4, 5, true, (void**)&dx));
  RMI_TRY(rmi_scratch(ctx, 0, m * n, (void**)&dq));
  RMI_TRY(rmi_scratch(ctx, 1, m * (n / 32) * 4, (void**)&ds));
  RMI_TRY(rmi_scratch(ctx, 6, m * w->n_rows * 4, (void**)&dout));
  RMI_TRY(launch_q8_quantize(ctx, dx, m, n, dq, ds, 0));
  RMI_TRY(launch_q4_0_matmul(ctx, w, dq, ds, m, dout, 0, w->n_rows));
  return host_out(ctx, output, dout, 1, m * w->n_rows * 4, 0);
}

// ---------------------------------------------------------------- embedding lookup

extern "C" int32_t rmi_embedding_lookup(rmi_ctx* ctx, const rmi_weight* w, const uint32_t* token_ids, size_t m,
                                        float* output) {
  RMI_TRY(rmi_check_ctx(ctx));
  RMI_TRY(rmi_check_weight(w, -1));
  RMI_REQUIRE(w->ggml_type == RMI_GGML_Q8_0 || w->ggml_type == RMI_GGML_Q4_0 || w->ggml_type == RMI_GGML_Q6_K,
              RMI_ERR_UNSUPPORTED, "unsupported embedding type %d (Q8_0, Q4_0 and Q6_K are handled)", w->ggml_type);
  if (m == 0 || w->n_in == 0) return RMI_OK;
  RMI_REQUIRE(token_ids && output, RMI_ERR_BAD_HANDLE, "rmi_embedding_lookup: null buffer");
  for (size_t i = 0; i < m; i++)
    RMI_REQUIRE(token_ids[i] < w->n_rows, RMI_ERR_BAD_SHAPE, "token id %u at position %zu is outside the table of %zu rows",
                token_ids[i], i, w->n_rows);
  std::lock_guard<std::mutex> lock(ctx->mu);
  uint32_t* dids;
  float* dout;
  RMI_TRY(rmi_scratch(ctx, 0, m * 4, (void**)&dids));
  RMI_TRY(rmi_scratch(ctx, 6, m * w->n_in * 4, (void**)&dout));
  RMI_CUDA_CHECK(cudaMemcpyAsync(dids, token_ids, m * 4, cudaMemcpyHostToDevice, ctx->stream));
  if (w->ggml_type == RMI_GGML_Q8_0) RMI_TRY(launch_q8_embedding(ctx, w, dids, m, dout));
  else if (w->ggml_type == RMI_GGML_Q4_0) RMI_TRY(launch_q4_0_embedding(ctx, w, dids, m, dout));
  else RMI_TRY(launch_q6k_embedding(ctx, w, dids, m, dout));
  RMI_CUDA_CHECK(cudaMemcpyAsync(output, dout, m * w->n_in * 4, cudaMemcpyDeviceToHost, ctx->stream));
  RMI_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
  return RMI_OK;
}
