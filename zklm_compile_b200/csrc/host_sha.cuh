// SHA-256 over bytes that are in host memory anyway, by the calling thread.
//
// A hash chain is serial, and a lone GPU thread takes 0.87 us a block (64 dependent rounds at 27 cycles); a CPU core with the SHA
// instructions takes 0.05 us, one without them 0.3.  So a caller's transcript that absorbs a long vector which the
// call has on the host (the scores and outputs of a row attention proof: read from it, or written into it) absorbs it here: its
// 112-byte state is fetched, advanced and put back in stream order.
#pragma once
#include "context.cuh"
#include <cstring>
#if defined(__x86_64__)
#include <cpuid.h>
#include <immintrin.h>
#endif

namespace zkb {

static const u32 SHA_K_HOST[64] = {
    0x428a2f98, 0x71374491, 0xb5c0fbcf, 0xe9b5dba5, 0x3956c25b, 0x59f111f1, 0x923f82a4, 0xab1c5ed5,
    0xd807aa98, 0x12835b01, 0x243185be, 0x550c7dc3, 0x72be5d74, 0x80deb1fe, 0x9bdc06a7, 0xc19bf174,
    0xe49b69c1, 0xefbe4786, 0x0fc19dc6, 0x240ca1cc, 0x2de92c6f, 0x4a7484aa, 0x5cb0a9dc, 0x76f988da,
    0x983e5152, 0xa831c66d, 0xb00327c8, 0xbf597fc7, 0xc6e00bf3, 0xd5a79147, 0x06ca6351, 0x14292967,
    0x27b70a85, 0x2e1b2138, 0x4d2c6dfc, 0x53380d13, 0x650a7354, 0x766a0abb, 0x81c2c92e, 0x92722c85,
    0xa2bfe8a1, 0xa81a664b, 0xc24b8b70, 0xc76c51a3, 0xd192e819, 0xd6990624, 0xf40e3585, 0x106aa070,
    0x19a4c116, 0x1e376c08, 0x2748774c, 0x34b0bcb5, 0x391c0cb3, 0x4ed8aa4a, 0x5b9cca4f, 0x682e6ff3,
    0x748f82ee, 0x78a5636f, 0x84c87814, 0x8cc70208, 0x90befffa, 0xa4506ceb, 0xbef9a3f7, 0xc67178f2};

inline void sha256_blocks_plain(u32* st, const unsigned char* p, size_t blocks) {
    auto rotr = [](u32 x, int n) { return (x >> n) | (x << (32 - n)); };
    for (; blocks; blocks--, p += 64) {
        u32 w[64], s[8];
        for (int i = 0; i < 16; i++) w[i] = ((u32)p[4 * i] << 24) | ((u32)p[4 * i + 1] << 16) | ((u32)p[4 * i + 2] << 8) | p[4 * i + 3];
        for (int i = 16; i < 64; i++)
            w[i] = w[i - 16] + (rotr(w[i - 15], 7) ^ rotr(w[i - 15], 18) ^ (w[i - 15] >> 3)) + w[i - 7] + (rotr(w[i - 2], 17) ^ rotr(w[i - 2], 19) ^ (w[i - 2] >> 10));
        memcpy(s, st, 32);
        for (int i = 0; i < 64; i++) {
            const u32 t1 = s[7] + (rotr(s[4], 6) ^ rotr(s[4], 11) ^ rotr(s[4], 25)) + ((s[4] & s[5]) ^ (~s[4] & s[6])) + SHA_K_HOST[i] + w[i];
            const u32 t2 = (rotr(s[0], 2) ^ rotr(s[0], 13) ^ rotr(s[0], 22)) + ((s[0] & s[1]) ^ (s[0] & s[2]) ^ (s[1] & s[2]));
            for (int k = 7; k > 0; k--) s[k] = s[k - 1];
            s[4] += t1;
            s[0] = t1 + t2;
        }
        for (int i = 0; i < 8; i++) st[i] += s[i];
    }
}
#if defined(__x86_64__)
// The same with the CPU's SHA instructions: four rounds a pair of sha256rnds2, whose operands hold {a, b, e, f} and {c, d, g, h}.
__attribute__((target("sha,sse4.1,ssse3"))) inline void sha256_blocks_ni(u32* st, const unsigned char* p, size_t blocks) {
    const __m128i order = _mm_set_epi64x(0x0c0d0e0f08090a0bll, 0x0405060700010203ll);
    __m128i abef = _mm_set_epi32((int)st[0], (int)st[1], (int)st[4], (int)st[5]), cdgh = _mm_set_epi32((int)st[2], (int)st[3], (int)st[6], (int)st[7]);
    for (; blocks; blocks--, p += 64) {
        const __m128i abef0 = abef, cdgh0 = cdgh;
        __m128i m[4];
        for (int i = 0; i < 4; i++) m[i] = _mm_shuffle_epi8(_mm_loadu_si128(reinterpret_cast<const __m128i*>(p + 16 * i)), order);
        for (int i = 0; i < 16; i++) {           // words 4 i .. 4 i + 3 are in m[i & 3]
            const __m128i kw = _mm_add_epi32(m[i & 3], _mm_loadu_si128(reinterpret_cast<const __m128i*>(SHA_K_HOST + 4 * i)));
            cdgh = _mm_sha256rnds2_epu32(cdgh, abef, kw);
            abef = _mm_sha256rnds2_epu32(abef, cdgh, _mm_shuffle_epi32(kw, 0x0e));
            if (i < 12) {                        // words 4 (i + 4) .. take the place of the oldest four
                const __m128i w7 = _mm_alignr_epi8(m[(i + 3) & 3], m[(i + 2) & 3], 4);
                m[i & 3] = _mm_sha256msg2_epu32(_mm_add_epi32(_mm_sha256msg1_epu32(m[i & 3], m[(i + 1) & 3]), w7), m[(i + 3) & 3]);
            }
        }
        abef = _mm_add_epi32(abef, abef0);
        cdgh = _mm_add_epi32(cdgh, cdgh0);
    }
    u32 x[4], y[4];
    _mm_storeu_si128(reinterpret_cast<__m128i*>(x), abef);
    _mm_storeu_si128(reinterpret_cast<__m128i*>(y), cdgh);
    st[0] = x[3]; st[1] = x[2]; st[4] = x[1]; st[5] = x[0];
    st[2] = y[3]; st[3] = y[2]; st[6] = y[1]; st[7] = y[0];
}
inline bool cpu_has_sha() {
    unsigned a = 0, b = 0, c = 0, d = 0;
    if (!__get_cpuid(1, &a, &b, &c, &d) || !(c & bit_SSE4_1) || !(c & bit_SSSE3)) return false;
    return __get_cpuid_count(7, 0, &a, &b, &c, &d) && (b & (1u << 29));
}
#endif
inline void sha256_blocks_host(u32* st, const unsigned char* p, size_t blocks) {
#if defined(__x86_64__)
    static const bool ni = cpu_has_sha();
    if (ni) { sha256_blocks_ni(st, p, blocks); return; }
#endif
    sha256_blocks_plain(st, p, blocks);
}
// n bytes into a transcript's state (Transcript::absorb_bytes, sumcheck.rs:136-140).
inline void tr_absorb_host(TrState& t, const void* bytes, size_t n) {
    if (t.buflen > 63) throw ArgFail{ZKB_E_CUDA, "transcript state did not arrive"};
    const unsigned char* p = static_cast<const unsigned char*>(bytes);
    t.total += n;
    if (t.buflen) {
        const size_t m = n < 64 - (size_t)t.buflen ? n : 64 - (size_t)t.buflen;
        memcpy(t.buf + t.buflen, p, m);
        t.buflen += (u32)m; p += m; n -= m;
        if (t.buflen < 64) return;
        sha256_blocks_host(t.h, t.buf, 1);
        t.buflen = 0;
    }
    sha256_blocks_host(t.h, p, n / 64);
    memcpy(t.buf, p + (n & ~size_t(63)), n & 63);
    t.buflen = (u32)(n & 63);
}

// A long absorb of a caller's transcript on the host: begin() behind whatever advances the transcript, finish() once the words are here
// and the context's stream, on which begin() was enqueued, has been waited for.
// From HOST_ABSORB_MIN words on: on the device such a stream takes about as long as the wait and the two copies (and row proofs of that many
// words as long as either).  Measured on B200, device / host, us: a proof of 1280 words 348 / 362, of 1920 356 / 364, of 2448 376 / 382, of
// 2560 373 / 369, of 2880 396 / 372, of 4096 470 / 386; checks and op lists of such proofs cross there too.  Checking 1232 attention rows with
// a stream of 15 785 blocks 14.96 -> 2.06 ms.
constexpr size_t HOST_ABSORB_MIN = 2560;
struct HostAbsorb {
    zkb_ctx* const c;
    TrState* const dev;
    const bool on;
    HostAbsorb(zkb_ctx* ctx, TrState* tr, size_t words) : c(ctx), dev(tr), on(tr && words >= HOST_ABSORB_MIN && !ctx->capturing) {}
    void begin() const { if (on) ZKB_CUDA(cudaMemcpyAsync(c->transcript_host(), dev, sizeof(TrState), cudaMemcpyDeviceToHost, c->stream)); }
    void finish(const u32* head, size_t n_head, const u32* words, size_t n_words) const {
        TrState* t = c->transcript_host();
        tr_absorb_host(*t, head, n_head * 4);
        tr_absorb_host(*t, words, n_words * 4);
        ZKB_CUDA(cudaMemcpyAsync(dev, t, sizeof(TrState), cudaMemcpyHostToDevice, c->stream));
    }
};

}  // namespace zkb
