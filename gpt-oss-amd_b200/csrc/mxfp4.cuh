// MXFP4 kernels outside the GEMMs: exact unpack of checkpoint-layout tensors,
// re-tiling into the resident layout at upload, and a decode of resident
// weights through the GEMM's own decode function (for bit-exactness tests).
#pragma once
#include "common.cuh"

namespace moe {

// prmt with the sign-replicating selector bit (__byte_perm masks it out).
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// Checkpoint codes -> bf16, four at a time.  `sel` holds four e2m1 codes in its low 16 bits.
// A code s|e1 e0|m at bf16 bits 15, [8:6] is value * 2^-126 (common.cuh); its low byte (e0 m
// at bits 7:6) and its high byte (s at bit 7, e1 at bit 0) come from byte-permute lookups
// indexed by the codes themselves.  Selector bit 3 makes the permute replicate the byte's
// sign, which turns the sign of a code into 0x80 / 0xFF bytes.
__device__ __forceinline__ void mxfp4_codes_to_bf16(uint32_t sel, uint32_t out[2]) {
    const uint32_t mag = sel & 0x7777u;
    const uint32_t lo = prmt(0xC0804000u, 0xC0804000u, mag);
    const uint32_t e1 = prmt(0x00000000u, 0x01010101u, mag);
    const uint32_t sg = prmt(0x80808080u, 0x80808080u, sel);
    const uint32_t hi = ((sg << 1) & 0x80808080u) | e1;
    out[0] = prmt(lo, hi, 0x5140);
    out[1] = prmt(lo, hi, 0x7362);
}

// blocks [rows, G, 16] u8, scales [rows, G] u8 -> out [rows, 32*G] bf16 bits, for every scale
// byte.  The product of a code and a scale is exact in bf16 or overflows to infinity (byte
// 254 / 255), so it is one multiply by 2^(byte - 1), and for bytes above 128, where that
// is no bf16 number, a multiply by 2^127 and one by 2^(byte - 128).
//
// Bound by HBM: 17 B read, 64 B written per block of 32.  A thread decodes one 32-bit word
// into one 16-byte store, so a warp's loads and stores are whole consecutive lines, and it
// has UNPACK_WORDS words in flight.  Gate/up matrices of 32 experts at hidden 2880 (1.34 GB):
// 467 -> 211 us, 6.4 TB/s (before: a thread per block, its four stores 64 bytes apart from
// its neighbour's, and integer arithmetic element by element).
constexpr int UNPACK_THREADS = 256;
constexpr int UNPACK_WORDS = 4;

__global__ void __launch_bounds__(UNPACK_THREADS)
mxfp4_unpack_kernel(const uint32_t* __restrict__ words, const uint8_t* __restrict__ scales, long long n_words,
                    uint4* __restrict__ out) {
    const long long i0 = (long long)blockIdx.x * (UNPACK_THREADS * UNPACK_WORDS) + threadIdx.x;
    uint32_t w[UNPACK_WORDS], sb[UNPACK_WORDS];
#pragma unroll
    for (int u = 0; u < UNPACK_WORDS; u++) {
        const long long i = i0 + u * UNPACK_THREADS;
        w[u] = i < n_words ? __ldcs(words + i) : 0u;
        sb[u] = i < n_words ? scales[i >> 2] : 0u;  // four words per block
    }
#pragma unroll
    for (int u = 0; u < UNPACK_WORDS; u++) {
        const long long i = i0 + u * UNPACK_THREADS;
        uint32_t r[4];
        mxfp4_codes_to_bf16(w[u], r);
        mxfp4_codes_to_bf16(w[u] >> 16, r + 2);
        const uint32_t m = mxfp4_scale_mult(min(sb[u], (uint32_t)MAX_SCALE_BYTE));
#pragma unroll
        for (int p = 0; p < 4; p++)
            r[p] = bf16x2_mul(r[p], m);
        if (sb[u] > (uint32_t)MAX_SCALE_BYTE) {
            const uint32_t m2 = mxfp4_scale_mult(sb[u] - (uint32_t)MAX_SCALE_BYTE + 1u);
#pragma unroll
            for (int p = 0; p < 4; p++)
                r[p] = bf16x2_mul(r[p], m2);
        }
        if (i < n_words)
            __stcs(out + i, make_uint4(r[0], r[1], r[2], r[3]));
    }
}

// The GEMMs' one-multiply decode covers resident scale bytes 0..MAX_SCALE_BYTE.  A
// checkpoint may hold any e8m0 byte (the reference's dequantize_fp4 takes them all,
// tools/model_export/gpt-oss-20b/export_model_bin.py:125-129), so every weight ROW gets
// an exponent shift: shift = max(0, largest scale byte of the row - MAX_SCALE_BYTE), the
// resident bytes are the checkpoint's minus the shift, and the GEMM epilogue multiplies
// the row's fp32 accumulator by 2^shift (exact: a power of two).  A row is representable
// when the scale bytes of its blocks that hold a non-zero code span at most
// MAX_SCALE_BYTE binades; a row that does not is reported (DS_BAD_SCALE).  Blocks of
// zeros keep their zeros under any scale.
// One warp per row.  row_shift[rows] (ints, scratch for the re-tile kernel that follows
// on the same stream) and row_scale[rows] = 2^shift.
__global__ void mxfp4_row_shift_kernel(const uint8_t* __restrict__ blocks,
                                       const uint8_t* __restrict__ scales, int rows, int G,
                                       int* __restrict__ row_shift, float* __restrict__ row_scale,
                                       int* __restrict__ status) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows)
        return;
    int hi = 0, lo = 255;
    for (int g = lane; g < G; g += 32) {
        const uint4 q = *reinterpret_cast<const uint4*>(blocks + ((size_t)row * G + g) * 16);
        if (((q.x | q.y | q.z | q.w) & 0x77777777u) != 0) {  // some magnitude is not zero
            const int sb = scales[(size_t)row * G + g];
            hi = max(hi, sb);
            lo = min(lo, sb);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    }
    if (lane == 0) {
        const int shift = max(0, hi - MAX_SCALE_BYTE);
        if (lo < shift)
            report_status(status, DS_BAD_SCALE);
        row_shift[row] = shift;
        row_scale[row] = __uint_as_float((uint32_t)(127 + shift) << 23);
    }
}

// Checkpoint layout of ONE expert matrix -> resident chunks.
// grid (k_stages, m_tiles), block TILE_M threads (thread = row of the tile).
__global__ void mxfp4_retile_kernel(const uint8_t* __restrict__ blocks,
                                    const uint8_t* __restrict__ scales, int rows, int G,
                                    const int* __restrict__ row_shift, uint8_t* __restrict__ chunks) {
    const int ks = blockIdx.x, mt = blockIdx.y, r = threadIdx.x;
    const int row = mt * TILE_M + r;
    const int shift = row < rows ? row_shift[row] : 0;
    uint8_t* chunk = chunks + ((size_t)mt * gridDim.x + ks) * CHUNK_BYTES;
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const int g = ks * 2 + b;
        uint4 q = make_uint4(0, 0, 0, 0);
        int sb = 127;
        if (row < rows && g < G) {
            q = *reinterpret_cast<const uint4*>(blocks + ((size_t)row * G + g) * 16);
            // only a block of zeros can leave the range (mxfp4_row_shift_kernel checked the rest)
            sb = min(max((int)scales[(size_t)row * G + g] - shift, 0), MAX_SCALE_BYTE);
        }
        q.x = mxfp4_retile_word(q.x);
        q.y = mxfp4_retile_word(q.y);
        q.z = mxfp4_retile_word(q.z);
        q.w = mxfp4_retile_word(q.w);
        *reinterpret_cast<uint4*>(chunk + b * PLANE_BYTES + r * 16) = q;
        chunk[2 * PLANE_BYTES + r * 2 + b] = (uint8_t)sb;
    }
}

// Resident chunks of one expert matrix -> row-major bf16 [rows, K] through
// mxfp4_decode_word, the function the GEMM main loops call, times the row's 2^shift
// (what the GEMM epilogue applies to the accumulator).
// grid (k_stages, m_tiles), block TILE_M threads.
__global__ void mxfp4_unpack_resident_kernel(const uint8_t* __restrict__ chunks,
                                             const float* __restrict__ row_scale, int rows, int K,
                                             uint16_t* __restrict__ out) {
    const int ks = blockIdx.x, mt = blockIdx.y, r = threadIdx.x;
    const int row = mt * TILE_M + r;
    if (row >= rows)
        return;
    const float rs = row_scale[row];
    const uint8_t* chunk = chunks + ((size_t)mt * gridDim.x + ks) * CHUNK_BYTES;
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const int col0 = ks * KSTAGE + b * 32;
        if (col0 >= K)
            continue;
        const uint4 q = *reinterpret_cast<const uint4*>(chunk + b * PLANE_BYTES + r * 16);
        const uint32_t mult = mxfp4_scale_mult(chunk[2 * PLANE_BYTES + r * 2 + b]);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        uint4* o = reinterpret_cast<uint4*>(out + (size_t)row * K + col0);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint32_t d[4];
            mxfp4_decode_word(w[j], mult, d);
            if (rs != 1.f) {
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    const float lo = __uint_as_float(d[p] << 16) * rs;
                    const float hi = __uint_as_float(d[p] & 0xFFFF0000u) * rs;
                    d[p] = pack_bf16x2(lo, hi);
                }
            }
            o[j] = make_uint4(d[0], d[1], d[2], d[3]);
        }
    }
}

}  // namespace moe
