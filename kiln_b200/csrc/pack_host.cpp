// AVX-512 form of the host packer's inner work (repack.cu: kiln_w4a16_quantize_and_pack_host), picked at run time.
//
// Bound: memory (a weight read, its dequantised value and half a byte written) once the arithmetic is vectorised.  The scalar
// loops spent 19 of 22 ms on a 2560 x 4096 weight (8 cores) on a division, a roundf call and per-nibble byte traffic for each
// weight; here sixteen columns are divided, rounded half away from zero and packed at a time.  Work is dealt in blocks of one
// scale group x 256 columns, 1 KB of every row, so that a block stays in a core's L2 between its two passes (maxima, then
// quantise).  Measured on 8 cores: 2560 x 4096 f32 28 -> 7 ms, of which the
// first touch of the 47 MB of fresh outputs takes more than half (into reused ones 22.6 -> 2.4 ms); on 16: 3.3 ms, 0.9 into reused ones
#include "pack_host.h"

#if defined(__x86_64__)
#include <immintrin.h>

#define KILN_AVX512 __attribute__((target("avx512f,avx512bw,avx512vl,avx512dq,f16c")))

namespace kiln {
namespace {

// max |w| of each column over `rows` rows (NaN never wins, as in the reference's comparison)
KILN_AVX512 void column_max(const float *w, size_t n, int rows, int cols, float *mx) {
    for (int c = 0; c < cols; c += 64) {
        __m512 m[4] = {_mm512_setzero_ps(), _mm512_setzero_ps(), _mm512_setzero_ps(), _mm512_setzero_ps()};
        for (int r = 0; r < rows; ++r) {
            const float *p = w + static_cast<size_t>(r) * n + c;
            for (int v = 0; v < 4; ++v) m[v] = _mm512_max_ps(_mm512_abs_ps(_mm512_loadu_ps(p + 16 * v)), m[v]);  // (NaN first: the second operand)
        }
        for (int v = 0; v < 4; ++v) _mm512_storeu_ps(mx + c + 16 * v, m[v]);
    }
}

// Quantised weight 0..15 of sixteen columns, and its dequantised value.
KILN_AVX512 inline __m512i quantize16(__m512 w, __m512 s, __m512 *dequant) {
    const __m512 q = _mm512_div_ps(w, s);
    const __m512 t = _mm512_roundscale_ps(q, _MM_FROUND_TO_ZERO | _MM_FROUND_NO_EXC);
    const __m512 d = _mm512_sub_ps(q, t);  // exact; half away from zero: one step out where it is at least one half
    const __mmask16 up = _mm512_cmp_ps_mask(_mm512_abs_ps(d), _mm512_set1_ps(0.5f), _CMP_GE_OQ);
    const __m512 one = _mm512_or_ps(_mm512_and_ps(q, _mm512_set1_ps(-0.0f)), _mm512_set1_ps(1.0f));
    __m512 r = _mm512_mask_add_ps(t, up, t, one);
    r = _mm512_min_ps(_mm512_max_ps(r, _mm512_set1_ps(-8.0f)), _mm512_set1_ps(7.0f));
    const __m512i qi = _mm512_cvtps_epi32(_mm512_maskz_mov_ps(_mm512_cmp_ps_mask(q, q, _CMP_ORD_Q), r));  // (NaN: 0)
    *dequant = _mm512_mul_ps(_mm512_cvtepi32_ps(qi), s);
    return _mm512_add_epi32(qi, _mm512_set1_epi32(8));
}

}  // namespace

bool pack_host_vectorised() { return __builtin_cpu_supports("avx512f") && __builtin_cpu_supports("avx512bw") && __builtin_cpu_supports("avx512vl") && __builtin_cpu_supports("avx512dq") && __builtin_cpu_supports("f16c"); }

// Rows [row0, row0 + rows) x columns [col0, col0 + cols) of the [., n] weight: one scale group.  rows % 16 == 0, cols % 64 == 0.
KILN_AVX512 void pack_host_block(const float *weight, int n, int row0, int rows, int col0, int cols, int32_t *b_packed,
                                 uint16_t *scale_row, const int *scale_pos, float *dequant) {
    alignas(64) float mx[kHostBlockCols], sc[kHostBlockCols];
    alignas(64) uint16_t half[kHostBlockCols];
    const size_t row_words = static_cast<size_t>(2) * n;
    const float *w = weight + static_cast<size_t>(row0) * n + col0;
    column_max(w, n, rows, cols, mx);
    for (int c = 0; c < cols; c += 16) {
        __m512 m = _mm512_load_ps(mx + c);
        m = _mm512_mask_mov_ps(m, _mm512_cmp_ps_mask(m, _mm512_setzero_ps(), _CMP_EQ_OQ), _mm512_set1_ps(1.0f));
        const __m256i h = _mm512_cvtps_ph(_mm512_div_ps(_mm512_mul_ps(_mm512_set1_ps(2.0f), m), _mm512_set1_ps(15.0f)),
                                          _MM_FROUND_TO_NEAREST_INT | _MM_FROUND_NO_EXC);
        _mm256_store_si256(reinterpret_cast<__m256i *>(half + c), h);
        _mm512_store_ps(sc + c, _mm512_cvtph_ps(h));
    }
    for (int c = 0; c < cols; ++c) scale_row[col0 + (c & ~63) + scale_pos[c & 63]] = half[c];

    const __m512i idx = _mm512_mullo_epi32(_mm512_set_epi32(15, 14, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2, 1, 0), _mm512_set1_epi32(8));
    for (int kt = 0; kt < rows; kt += 16)
        for (int ch = 0; ch < cols; ch += 64) {
            // words[qd * 4 + j][c]: the word of lane (c, qd) and 16-column tile j
            alignas(64) uint32_t words[16][8];
            for (int j = 0; j < 4; ++j) {
                const int c = ch + 16 * j;
                const __m512 s = _mm512_load_ps(sc + c);
                for (int qd = 0; qd < 4; ++qd) {
                    static const int kRow[4] = {0, 8, 1, 9}, kShift[4] = {0, 4, 16, 20};
                    __m512i half_words = _mm512_setzero_si512();
                    for (int i = 0; i < 4; ++i) {
                        const size_t off = static_cast<size_t>(kt + 2 * qd + kRow[i]) * n + c;
                        __m512 dq;
                        const __m512i q = quantize16(_mm512_loadu_ps(w + off), s, &dq);
                        if (dequant) _mm512_storeu_ps(dequant + static_cast<size_t>(row0) * n + col0 + off, dq);
                        half_words = _mm512_or_si512(half_words, _mm512_slli_epi32(q, kShift[i]));
                    }
                    // columns c + 8 are nibbles 2, 3, 6, 7 of the words of columns c
                    const __m256i lo = _mm512_castsi512_si256(half_words), hi = _mm512_extracti64x4_epi64(half_words, 1);
                    _mm256_store_si256(reinterpret_cast<__m256i *>(words[qd * 4 + j]), _mm256_or_si256(lo, _mm256_slli_epi32(hi, 8)));
                }
            }
            int32_t *out = b_packed + static_cast<size_t>((row0 + kt) / 16) * row_words + static_cast<size_t>(col0 + ch) * 2;
            for (int c = 0; c < 8; ++c)
                _mm512_storeu_si512(out + 16 * c, _mm512_i32gather_epi32(idx, reinterpret_cast<const int *>(&words[0][c]), 4));
        }
}

}  // namespace kiln

#else

namespace kiln {
bool pack_host_vectorised() { return false; }
void pack_host_block(const float *, int, int, int, int, int, int32_t *, uint16_t *, const int *, float *) {}
}  // namespace kiln

#endif
