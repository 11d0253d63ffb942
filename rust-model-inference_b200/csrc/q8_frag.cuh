// Operand layouts of the tensor-core Q8_0 matmul in the eight-lane order (q8_mma.cu): a thread's share of an MMA operand
// is one aligned piece of a record, so it costs one shared-memory load and no data movement.
//
// A 32-block of a row has eight words of four bytes; word L = bytes 4L..4L+3 belongs to lane L of the reference's AVX2
// accumulator.  The block is dealt to the four threads c of an MMA row: thread c owns bytes 2h, 2h+1 (h = c % 2) of the
// words 4l + j, j = 0..3 (l = c / 2).  MMA j (f16 m16n8k8) multiplies words j (threads 0, 1) and 4 + j (threads 2, 3);
// the columns of the other operand hold one of the two words and zeros in the place of the other, so the two columns of
// an activation row are its partial sums of the lanes j and 4 + j.
//
// Weight records (16 rows x 32 values, 544 bytes): 16 f16 scales as (row r, row r + 8) pairs, then 32 threads x 16 bytes
// (row r: j = 0, 1 | row r + 8: j = 0, 1 | row r: j = 2, 3 | row r + 8: j = 2, 3).
// Activation records (4 rows x 32 values, 272 bytes): 16 slots x 16 bytes, slot = row * 4 + c, f16 pairs by j; then the
// four f32 scales.
// The records that one CTA needs of a block lie together, block after block: [tile / 4][block][tile % 4] for weights,
// [group / 2^pack][block][group % 2^pack] for activations.
#pragma once
#include "common.cuh"

static constexpr int FRAG_W_REC = 544, FRAG_W_PACK = 4;
static constexpr int FRAG_X_REC = 272;

// Where the quantizers put their result.
struct q8_dst {
  uint8_t* q8;    // row-major [m][n] bytes, or records
  float* scales;  // row-major [m][n / 32]; null for records
  int pack;       // records: log2 of the activation groups that lie together; -1: row-major
};

inline size_t frag_w_bytes(size_t n_tiles16, size_t blocks) {
  return (n_tiles16 + FRAG_W_PACK - 1) / FRAG_W_PACK * FRAG_W_PACK * blocks * FRAG_W_REC;
}
// for every pack up to 2^4
inline size_t frag_x_bytes(size_t m, size_t blocks) { return (m + 63) / 64 * 16 * blocks * FRAG_X_REC; }

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t frag_pair(int lo, int hi) {
  const __half2 h = __floats2half2_rn((float)lo, (float)hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint8_t* frag_x_record(const q8_dst& d, size_t blocks, size_t t, size_t b) {
  const size_t g = t >> 2;
  return d.q8 + ((((g >> d.pack) * blocks + b) << d.pack) + (g & ((1u << d.pack) - 1))) * FRAG_X_REC;
}
// One quantized value: byte i of block b of row t.
__device__ __forceinline__ void store_q8_value(const q8_dst& d, size_t blocks, size_t t, size_t b, int i, int q) {
  if (d.pack < 0) {
    d.q8[(t * blocks + b) * 32 + i] = (uint8_t)(int8_t)q;
  } else {
    const int l = i >> 4, j = (i >> 2) & 3, h = (i >> 1) & 1;
    *reinterpret_cast<__half*>(frag_x_record(d, blocks, t, b) + ((t & 3) * 4 + l * 2 + h) * 16 + j * 4 + (i & 1) * 2) = __int2half_rn(q);
  }
}
// The four values of word L; rows on a 4-byte boundary.
__device__ __forceinline__ void store_q8_word(const q8_dst& d, size_t blocks, size_t t, size_t b, int L, int q0, int q1, int q2, int q3) {
  if (d.pack < 0) {
    *reinterpret_cast<uint32_t*>(d.q8 + (t * blocks + b) * 32 + 4 * L) =
        (uint32_t)(q0 & 0xff) | (uint32_t)(q1 & 0xff) << 8 | (uint32_t)(q2 & 0xff) << 16 | (uint32_t)(q3 & 0xff) << 24;
  } else {
    uint8_t* p = frag_x_record(d, blocks, t, b) + ((t & 3) * 4 + (L >> 2) * 2) * 16 + (L & 3) * 4;
    *reinterpret_cast<uint32_t*>(p) = frag_pair(q0, q1);
    *reinterpret_cast<uint32_t*>(p + 16) = frag_pair(q2, q3);
  }
}
__device__ __forceinline__ void store_q8_scale(const q8_dst& d, size_t blocks, size_t t, size_t b, float sc) {
  if (d.pack < 0) d.scales[t * blocks + b] = sc;
  else *reinterpret_cast<float*>(frag_x_record(d, blocks, t, b) + 256 + (t & 3) * 4) = sc;
}
#endif
