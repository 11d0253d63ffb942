// Q8_0 x Q8_0 matmul of several activation rows on the tensor cores, in the AVX2 order of the reference, bit for bit
// (src/ops/kernel/q8_0/avx2.rs:53-174): eight chains per output, chain L accumulates
// fma(wd * xs, f32(sum of the four products of word L), acc) over the 32-blocks, then hsum_ps (dot.rs:447-456).
//
// The order leaves an accumulator of the tensor core only four products to add, so the results of every MMA are consumed at
// once by fp32 instructions; warp-level MMAs deliver them to the registers of the threads that do.  f16 m16n8k8: bytes are
// exact in f16, a sum of four products is an exact f32 integer and needs no conversion, and the zero-filled columns
// (q8_frag.cuh) give two of the eight words per MMA.  Per 16 rows x 4 activation rows x 32 products: four MMAs (8 cycles
// each on a sub-partition's tensor pipe), 16 fused multiply-adds and 2 multiplies (about 21 cycles on its fp32 pipe); both
// together measured 41.  Scalar multiply-adds: a packed f32x2 one with three distinct operands takes 3.3 cycles, two
// scalar ones with a shared multiplier 2.3.
//
// Bound: instruction issue and MMA latency at two warps per sub-partition (tensor pipe 53 % busy, fp32 pipe 35 %).
// Measured, 6144 x 1024: 480 rows 82 us, 74 T products-and-sums/s (dp4a GEMV: 150 us); 32 rows 10.7 us (20).
//
// A CTA (four warps, one 16-row weight tile each) walks K in chunks through a ring of stages; the records that it needs of
// a chunk are one bulk copy for the weights and one for the activations, because every further copy costs the issuing
// thread a few hundred cycles.  CTAs are persistent and the ring runs on across tiles.
#include "common.cuh"
#include "kernels.cuh"
#include "mma_dev.cuh"
#include "q8_frag.cuh"

namespace {

constexpr int LANES_THREADS = 128;
// Four rows and fewer: one pass of the GEMV kernels, which quantize in the same launch where they can, is as fast
// (3 rows of 4096 x 4096: 14.1 us, here 15.8).  Five and more rows: here one pass whatever their number (5..8 rows of
// 151936 x 1024: 52 us, GEMV 67 to 100; 19 rows of 896 x 4864: 10 us, GEMV 17).
constexpr size_t LANES_MIN_M = 5;

struct lanes_params {
  const uint8_t* w;      // weight records [tile / 4][block][tile % 4]
  const uint8_t* x;      // activation records [group / TG][block][group % TG]
  int blocks;
  int n_tiles16;         // weight row tiles
  int tiles_t, n_tiles;  // CTA tiles along the activation rows, in all (activation rows run fastest)
  int m, n_rows;
  float* out;            // [m][out_stride]
  size_t out_stride;
  rmi_dev_status* status;
  out_fanout fo;
};

// Stages of KC blocks; the refilled stage is that of the item LAG before the current one, so that with four stages the
// feeding thread does not wait for the slowest warp.
template <int TG, int KC, int S>
struct lanes_ring {
  static_assert(S <= 7, "barriers");
  static constexpr int W_BLOCK = FRAG_W_PACK * FRAG_W_REC, X_BLOCK = TG * FRAG_X_REC;
  static constexpr int B0 = KC * W_BLOCK, STAGE = B0 + KC * X_BLOCK, SMEM = 128 + S * STAGE;
  int tile, chunk;  // the next item
  __device__ __forceinline__ void copy_w(const lanes_params& p, uint32_t smem, int st, int nb) const {
    const int tr = tile / p.tiles_t;
    bulk_load(smem + 128 + st * STAGE, p.w + ((size_t)tr * p.blocks + chunk * KC) * W_BLOCK, nb * W_BLOCK, smem + 8 * st);
  }
  __device__ __forceinline__ void copy_x(const lanes_params& p, uint32_t smem, int st, int nb) const {
    const int tt = tile % p.tiles_t;
    bulk_load(smem + 128 + st * STAGE + B0, p.x + ((size_t)tt * p.blocks + chunk * KC) * X_BLOCK, nb * X_BLOCK, smem + 8 * st);
  }
  __device__ __forceinline__ void advance(int n_chunks) {
    if (++chunk == n_chunks) chunk = 0, tile += gridDim.x;
  }
  // The first S items; the weights' part travels before the wait on the preceding kernel, which writes activations only.
  __device__ __forceinline__ void start(const lanes_params& p, uint32_t smem, int n_chunks) {
    for (int pass = 0; pass < 2; pass++) {
      if (pass == 1) pdl_wait();
      tile = blockIdx.x, chunk = 0;
      for (int st = 0; st < S && tile < p.n_tiles; st++) {
        const int nb = min(KC, p.blocks - chunk * KC);
        if (pass == 0) {
          mbar_expect_tx(smem + 8 * st, nb * (W_BLOCK + X_BLOCK));
          copy_w(p, smem, st, nb);
        } else {
          copy_x(p, smem, st, nb);
        }
        advance(n_chunks);
      }
    }
  }
  // Item `item`, once every warp has released its stage.
  __device__ __forceinline__ void next(const lanes_params& p, uint32_t smem, int n_chunks, int item, int* abort_flag) {
    if (tile >= p.n_tiles) return;
    const int st = item % S, nb = min(KC, p.blocks - chunk * KC);
    if (!mbar_wait(smem + 64 + 8 * st, ((item / S) & 1) ^ 1, abort_flag, p.status, 12, item)) return;
    mbar_expect_tx(smem + 8 * st, nb * (W_BLOCK + X_BLOCK));
    copy_w(p, smem, st, nb);
    copy_x(p, smem, st, nb);
    advance(n_chunks);
  }
};

// A CTA tile is 64 weight rows (one 16-row tile per warp) x 4 TG activation rows.
template <int TG, int KC, int S, int MINB>
__global__ void __launch_bounds__(LANES_THREADS, MINB) q8_mma_lanes_kernel(const lanes_params p) {
  constexpr int LAG = S > 3 ? 2 : 1;
  using ring_t = lanes_ring<TG, KC, S>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const uint32_t smem = smem_u32(smem_raw);
  int* abort_flag = reinterpret_cast<int*>(smem_raw + 120);
  if (threadIdx.x == 0) {
    for (int i = 0; i < S; i++) {
      mbar_init(smem + 8 * i, 1);
      mbar_init(smem + 64 + 8 * i, 4);
    }
    *abort_flag = 0;
    mbar_init_fence();
  }
  __syncthreads();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_chunks = (p.blocks + KC - 1) / KC;
  ring_t ring;
  if (threadIdx.x == 0) ring.start(p, smem, n_chunks);
  __syncwarp();
  pdl_wait();
  const int r = lane >> 2, c = lane & 3;
  // this lane's operand slot: column (row lane / 8 of the group, word half (lane / 4) % 2), k positions of thread c
  const int lhalf = r & 1;
  const int live = (c >> 1) == lhalf;
  const uint8_t* a_base = smem_raw + 128 + warp * FRAG_W_REC;
  const uint8_t* b_base = smem_raw + 128 + ring_t::B0;
  const uint32_t slot = ((lane >> 3) * 4 + lhalf * 2 + (c & 1)) * 16;
  uint32_t b[2][4];  // operand registers of two groups; lanes whose k positions belong to the other word keep zeros
#pragma unroll
  for (int u = 0; u < 2; u++)
#pragma unroll
    for (int i = 0; i < 4; i++) b[u][i] = 0u;

  int item = 0;
  for (int tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
    const int tr = tile / p.tiles_t, tt = tile - tr * p.tiles_t;
    const int rt = tr * FRAG_W_PACK + warp, t0 = tt * TG * 4;
    const bool busy = rt < p.n_tiles16 && t0 < p.m;
    float acc[TG][4][4];
#pragma unroll
    for (int g = 0; g < TG; g++)
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[g][j][e] = 0.0f;
    for (int ch = 0; ch < n_chunks; ch++, item++) {
      const int st = item % S;
      if (!mbar_wait(smem + 8 * st, (item / S) & 1, abort_flag, p.status, 13, item)) return;
      if (threadIdx.x == 0 && item >= LAG) ring.next(p, smem, n_chunks, item - LAG + S, abort_flag);
      __syncwarp();
      if (busy) {
        const uint8_t* ap = a_base + st * ring_t::STAGE;
        const uint8_t* bp = b_base + st * ring_t::STAGE;
        const int nb = min(KC, p.blocks - ch * KC);
        uint4 an = *reinterpret_cast<const uint4*>(ap + 32 + lane * 16);
        __half2 sn = *reinterpret_cast<const __half2*>(ap + r * 4);
#pragma unroll TG > 2 ? 1 : (TG > 1 ? 2 : 4)
        for (int kb = 0; kb < nb; kb++) {
          const uint4 aw = an;
          const float2 wd = __half22float2(sn);
          if (kb + 1 < nb) ap += ring_t::W_BLOCK;   // the next block's weights while this one is multiplied
          an = *reinterpret_cast<const uint4*>(ap + 32 + lane * 16);
          sn = *reinterpret_cast<const __half2*>(ap + r * 4);
          // signed bytes to f16: 0x6400 | (q + 128) is 1152 + q
          uint32_t a[4][2];
          const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));
          const uint32_t wv[4] = {aw.x ^ 0x80808080u, aw.y ^ 0x80808080u, aw.z ^ 0x80808080u, aw.w ^ 0x80808080u};
#pragma unroll
          for (int j = 0; j < 4; j++)
#pragma unroll
            for (int half = 0; half < 2; half++) {
              const uint32_t v = __byte_perm(wv[(j >> 1) * 2 + half], 0x64646464u, (j & 1) ? 0x4342u : 0x4140u);
              const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&v), bias);
              a[j][half] = *reinterpret_cast<const uint32_t*>(&h);
            }
          float d[2][4][4], s[2][2];
#pragma unroll
          for (int g = 0; g <= TG; g++) {   // the MMAs of a group are issued before the results of the previous one are used
            if (g < TG) {
              asm volatile(
                  "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
                  "@p ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                  : "+r"(b[g & 1][0]), "+r"(b[g & 1][1]), "+r"(b[g & 1][2]), "+r"(b[g & 1][3])
                  : "r"(smem_u32(bp) + g * FRAG_X_REC + slot), "r"(live));
              const float xs = *reinterpret_cast<const float*>(bp + g * FRAG_X_REC + 256 + c * 4);
              s[g & 1][0] = __fmul_rn(wd.x, xs);
              s[g & 1][1] = __fmul_rn(wd.y, xs);
#pragma unroll
              for (int j = 0; j < 4; j++) mma_f16_k8(d[g & 1][j], a[j][0], a[j][1], b[g & 1][j]);
            }
            if (g > 0) {
#pragma unroll
              for (int j = 0; j < 4; j++)
#pragma unroll
                for (int e = 0; e < 4; e++)   // avx2.rs:96-148, lanes j and 4 + j
                  acc[g - 1][j][e] = __fmaf_rn(s[(g - 1) & 1][e >> 1], d[(g - 1) & 1][j][e], acc[g - 1][j][e]);
            }
          }
          bp += ring_t::X_BLOCK;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem + 64 + 8 * st);
    }
    if (!busy) continue;
#pragma unroll
    for (int g = 0; g < TG; g++) {
      const int t = t0 + 4 * g + c;
#pragma unroll
      for (int half = 0; half < 2; half++) {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++)  // dot.rs:447-456: s_i = a[i+4] + a[i]; (s0 + s1) + (s2 + s3)
          v[j] = __fadd_rn(acc[g][j][2 * half + 1], acc[g][j][2 * half]);
        const int row = rt * 16 + r + 8 * half;
        if (t < p.m && row < p.n_rows)
          store_fanout(p.out + (size_t)t * p.out_stride + row, __fadd_rn(__fadd_rn(v[0], v[1]), __fadd_rn(v[2], v[3])), p.fo);
      }
    }
  }
}

constexpr int MAX_DEVICES = 16;  // entries of the per-device occupancy caches

template <int TG, int KC, int S, int MINB>
int32_t run_lanes(rmi_ctx* ctx, lanes_params& p) {
  constexpr size_t smem = lanes_ring<TG, KC, S>::SMEM;
  auto kern = q8_mma_lanes_kernel<TG, KC, S, MINB>;
  static int cache[MAX_DEVICES];
  int& per_sm = cache[ctx->device % MAX_DEVICES];
  if (per_sm == 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, LANES_THREADS, smem);
    if (e != cudaSuccess || per_sm < 1) {
      rmi_set_error("q8_mma_lanes needs %zu B of shared memory: %s", smem, cudaGetErrorString(e));
      return RMI_ERR_CUDA;
    }
  }
  p.tiles_t = (p.m + 4 * TG - 1) / (4 * TG);
  p.n_tiles = (p.n_tiles16 + FRAG_W_PACK - 1) / FRAG_W_PACK * p.tiles_t;
  const int slots = ctx->sm_count * per_sm;
  return rmi_run(ctx, "q8_mma_lanes", kern, dim3((unsigned)(p.n_tiles < slots ? p.n_tiles : slots)), dim3(LANES_THREADS), smem, p);
}

// tile16 -> weight records, one thread per (row tile, block, lane); tiles past the last are zeros.
__global__ void q8_lanes_build_kernel(const uint8_t* __restrict__ t16, uint8_t* __restrict__ dst, size_t n_tiles16, size_t n_packed,
                                      size_t blocks) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_packed * blocks * 32) return;
  const int lane = (int)(idx & 31), r = lane >> 2, c = lane & 3, l = c >> 1, h = c & 1;
  const size_t b = (idx >> 5) % blocks, tile = (idx >> 5) / blocks;
  uint8_t* rec = dst + ((tile / FRAG_W_PACK * blocks + b) * FRAG_W_PACK + tile % FRAG_W_PACK) * FRAG_W_REC;
  uint32_t w[2][2] = {}, sc = 0;
  if (tile < n_tiles16) {
    const uint8_t* src = t16 + (tile * blocks + b) * Q8_REC_BYTES;
    for (int half = 0; half < 2; half++) {
      const int row = r + 8 * half;
      sc |= (uint32_t)*reinterpret_cast<const uint16_t*>(src + 2 * row) << (16 * half);
      for (int j = 0; j < 4; j++)
        w[half][j >> 1] |= (uint32_t)*reinterpret_cast<const uint16_t*>(src + 32 + 32 * row + 4 * (4 * l + j) + 2 * h) << (16 * (j & 1));
    }
  }
  *reinterpret_cast<uint4*>(rec + 32 + lane * 16) = make_uint4(w[0][0], w[1][0], w[0][1], w[1][1]);
  if (c == 0) *reinterpret_cast<uint32_t*>(rec + r * 4) = sc;
}

int32_t ensure_lanes_layout(rmi_ctx* ctx, const rmi_weight* cw) {
  rmi_weight* w = const_cast<rmi_weight*>(cw);
  const size_t blocks = w->n_in / 32, bytes = frag_w_bytes(w->n_tiles16, blocks);
  uint8_t* d = nullptr;
  if (cudaMalloc((void**)&d, bytes ? bytes : 16) != cudaSuccess) {
    (void)cudaGetLastError();
    return RMI_ERR_OOM;
  }
  const size_t n_packed = (w->n_tiles16 + FRAG_W_PACK - 1) / FRAG_W_PACK * FRAG_W_PACK, n = n_packed * blocks * 32;
  q8_lanes_build_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(w->d_tile16, d, w->n_tiles16, n_packed, blocks);
  // complete before any kernel of a dependent launch may fetch it ahead of its wait
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
    cudaFree(d);
    return RMI_ERR_CUDA;
  }
  w->d_lanes = d;
  w->frag_bytes += bytes;
  return RMI_OK;
}

// Which tile for n_tiles16 weight row tiles and m activation rows: rounds of CTA tiles x the time of a round, measured
// for K = 1024 (us).  Few tiles want small ones (every SM takes part), many want large ones (the conversion of the weight
// bytes and the copies are shared by more activation rows).
struct lanes_choice {
  int pack;      // log2 of the activation groups of a CTA tile
  int per_sm;    // resident CTAs per SM
  float round_us;
};
constexpr lanes_choice LANES[] = {{0, 1, 3.2f}, {0, 2, 4.4f}, {1, 2, 5.6f}, {2, 2, 9.2f}, {3, 1, 9.0f}, {3, 2, 16.3f}};

int choose_lanes(const rmi_ctx* ctx, const rmi_weight* w, size_t m) {
  int best = 0;
  float best_us = 0.0f;
  for (int i = 0; i < (int)(sizeof LANES / sizeof LANES[0]); i++) {
    const size_t rows = (size_t)4 << LANES[i].pack, slots = (size_t)ctx->sm_count * LANES[i].per_sm;
    const size_t tiles = (w->n_tiles16 + FRAG_W_PACK - 1) / FRAG_W_PACK * ((m + rows - 1) / rows);
    const float us = (float)((tiles + slots - 1) / slots) * LANES[i].round_us;
    if (i == 0 || us < best_us) best = i, best_us = us;
  }
  return best;
}

}  // namespace

// The records are built on first use.  Inside a stream capture, or without memory for them, the GEMV kernels run: the
// results are the same bits.
int q8_lanes_pack(rmi_ctx* ctx, const rmi_weight* w, size_t m) {
  if (ctx->sem != RMI_SEM_AVX2 || m < LANES_MIN_M || w->n_rows == 0 || w->n_in == 0) return -1;
  if (w->d_lanes == nullptr) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
      (void)cudaGetLastError();
      return -1;
    }
    if (ensure_lanes_layout(ctx, w) != RMI_OK) return -1;
  }
  return LANES[choose_lanes(ctx, w, m)].pack;
}

int32_t launch_q8_rows(rmi_ctx* ctx, const rmi_weight* w, const q8_dst& x, size_t m, float* out, size_t out_stride) {
  if (x.pack < 0) return launch_q8_gemv(ctx, w, x.q8, x.scales, m, out, out_stride, 0, w->n_rows);
  lanes_params p = {};
  p.w = w->d_lanes;
  p.x = x.q8;
  p.blocks = (int)(w->n_in / 32);
  p.n_tiles16 = (int)w->n_tiles16;
  p.m = (int)m;
  p.n_rows = (int)w->n_rows;
  p.out = out;
  p.out_stride = out_stride;
  p.status = ctx->d_status;
  p.fo = ctx->fanout;
  switch (choose_lanes(ctx, w, m)) {
    case 0: return run_lanes<1, 16, 4, 1>(ctx, p);
    case 1: return run_lanes<1, 16, 2, 2>(ctx, p);
    case 2: return run_lanes<2, 16, 2, 2>(ctx, p);
    case 3: return run_lanes<4, 16, 2, 2>(ctx, p);
    case 4: return run_lanes<8, 16, 2, 1>(ctx, p);
    default: return run_lanes<8, 12, 2, 2>(ctx, p);
  }
}
