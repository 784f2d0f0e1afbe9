// Device-resident Fiat-Shamir transcript: a SHA-256 stream that lives in global memory and is
// advanced by one thread, or by one warp with a second one beside it, of whichever kernel finishes a protocol step, so challenges never
// travel to the host.  Mirrors the reference `Transcript`
// (rust/zk_ml_prover/src/proving/sumcheck.rs:110-206):
//   new(label)      stream = label bytes
//   absorb(u32)     4 little-endian bytes; absorb_bytes(raw)
//   squeeze()       d = SHA-256(stream); stream := d; first of the four little-endian u64
//                   windows of d below 2^64 - 4, reduced mod p
//   squeeze_ef()    four squeezes -> (re c0, im c0, re c1, im c1)
#pragma once
#include "m31.cuh"

namespace zkb {

#ifdef ZKB_STAMP
// Experiment build only: start / end time stamps of the serial hash kernels, by transcript.
struct StampRec { const void* key; unsigned long long t0, t1; unsigned kind, smid; };
constexpr unsigned STAMP_CAP = 1u << 16;
__device__ StampRec g_stamps[STAMP_CAP];
__device__ unsigned g_stamp_n;
__device__ __forceinline__ unsigned long long stamp_now() { unsigned long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t; }
__device__ __forceinline__ void stamp_put(const void* key, unsigned kind, unsigned long long t0) {
    unsigned smid; asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    unsigned i = atomicAdd(&g_stamp_n, 1u);
    if (i < STAMP_CAP) g_stamps[i] = StampRec{key, t0, stamp_now(), kind, smid};
}
#define ZKB_STAMP_BEGIN unsigned long long stamp_t0 = stamp_now();
#define ZKB_STAMP_END(key, kind) do { if (threadIdx.x == 0) stamp_put(key, kind, stamp_t0); } while (0)
#else
#define ZKB_STAMP_BEGIN
#define ZKB_STAMP_END(key, kind) do { } while (0)
#endif


// Global-memory image of the stream.  `buf` holds the bytes not yet compressed.
struct TrState {
    u32 h[8];
    u32 buflen;      // 0..63
    u32 _pad;
    u64 total;       // bytes absorbed into the current SHA-256 stream
    unsigned char buf[64];
};

__constant__ u32 SHA_K[64] = {
    0x428a2f98, 0x71374491, 0xb5c0fbcf, 0xe9b5dba5, 0x3956c25b, 0x59f111f1, 0x923f82a4, 0xab1c5ed5,
    0xd807aa98, 0x12835b01, 0x243185be, 0x550c7dc3, 0x72be5d74, 0x80deb1fe, 0x9bdc06a7, 0xc19bf174,
    0xe49b69c1, 0xefbe4786, 0x0fc19dc6, 0x240ca1cc, 0x2de92c6f, 0x4a7484aa, 0x5cb0a9dc, 0x76f988da,
    0x983e5152, 0xa831c66d, 0xb00327c8, 0xbf597fc7, 0xc6e00bf3, 0xd5a79147, 0x06ca6351, 0x14292967,
    0x27b70a85, 0x2e1b2138, 0x4d2c6dfc, 0x53380d13, 0x650a7354, 0x766a0abb, 0x81c2c92e, 0x92722c85,
    0xa2bfe8a1, 0xa81a664b, 0xc24b8b70, 0xc76c51a3, 0xd192e819, 0xd6990624, 0xf40e3585, 0x106aa070,
    0x19a4c116, 0x1e376c08, 0x2748774c, 0x34b0bcb5, 0x391c0cb3, 0x4ed8aa4a, 0x5b9cca4f, 0x682e6ff3,
    0x748f82ee, 0x78a5636f, 0x84c87814, 0x8cc70208, 0x90befffa, 0xa4506ceb, 0xbef9a3f7, 0xc67178f2};

__device__ __forceinline__ u32 rotr32(u32 x, int n) { return __funnelshift_r(x, x, n); }
__device__ __forceinline__ u32 bswap32(u32 x) { return __byte_perm(x, 0, 0x0123); }

// One SHA-256 compression.  The chaining value travels in registers (by value), the message
// block is read from 16 little-endian words of shared memory and byte-swapped on the fly; the
// 64 rounds are fully unrolled with the working variables renamed instead of moved, and the
// message schedule is kept in a 16-register window.  One thread runs this; the rounds are a
// strict dependency chain, so the remaining lever is instruction count, not parallelism.
struct Sha8 { u32 v[8]; };

// One round.  The logic and shift pipe takes an instruction of a lone warp about every two cycles (measured on B200:
// eight independent lop3 or shf per iteration run at 2.0 - 2.2 cycles each, a dependent one at 4.4),
// so a compression is bound by its instruction count, not by the dependency chain: the boolean
// functions are single lop3 instructions, and the additions are written as multiply-adds by one in
// the association  x = h + kw + ch,  e' = x + d + s1,  a' = x + maj + s0 + s1,  which ptxas places
// best (30.6 cycles per round against 33.8 for the textbook form).
__device__ __forceinline__ u32 sha_xor3(u32 a, u32 b, u32 c) { u32 r; asm("lop3.b32 %0, %1, %2, %3, 0x96;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
__device__ __forceinline__ u32 sha_ch(u32 e, u32 f, u32 g) { u32 r; asm("lop3.b32 %0, %1, %2, %3, 0xCA;" : "=r"(r) : "r"(e), "r"(f), "r"(g)); return r; }
__device__ __forceinline__ u32 sha_maj(u32 a, u32 b, u32 c) { u32 r; asm("lop3.b32 %0, %1, %2, %3, 0xE8;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
__device__ __forceinline__ u32 sha_add(u32 a, u32 b) { u32 r; asm("mad.lo.u32 %0, %1, 1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
#define ZKB_SHA_RND(a, b, c, d, e, f, g, h, kw)                                   \
    {                                                                             \
        const u32 ch_ = sha_ch(e, f, g);                                          \
        const u32 mj_ = sha_maj(a, b, c);                                         \
        const u32 s1_ = sha_xor3(rotr32(e, 6), rotr32(e, 11), rotr32(e, 25));     \
        const u32 s0_ = sha_xor3(rotr32(a, 2), rotr32(a, 13), rotr32(a, 22));     \
        const u32 x_ = sha_add(sha_add(h, (kw)), ch_);                            \
        const u32 z_ = sha_add(x_, mj_);                                          \
        d = sha_add(sha_add(x_, d), s1_);                                         \
        h = sha_add(sha_add(z_, s0_), s1_);                                       \
    }
#define ZKB_SHA_SCHED(i) \
    (w[(i) & 15] += (rotr32(w[((i) + 1) & 15], 7) ^ rotr32(w[((i) + 1) & 15], 18) ^ (w[((i) + 1) & 15] >> 3)) + w[((i) + 9) & 15] + \
                    (rotr32(w[((i) + 14) & 15], 17) ^ rotr32(w[((i) + 14) & 15], 19) ^ (w[((i) + 14) & 15] >> 10)))

__device__ __noinline__ Sha8 sha256_compress(Sha8 hin, const u32* __restrict__ blk) {
    u32 w[16];
#pragma unroll
    for (int i = 0; i < 16; i++) w[i] = bswap32(blk[i]);
    u32 a = hin.v[0], b = hin.v[1], c = hin.v[2], d = hin.v[3], e = hin.v[4], f = hin.v[5], g = hin.v[6], h = hin.v[7];
#define ZKB_SHA_RND8(k0, i)                                                 \
    ZKB_SHA_RND(a, b, c, d, e, f, g, h, SHA_K[(k0) + (i)] + w[(i)]);         \
    ZKB_SHA_RND(h, a, b, c, d, e, f, g, SHA_K[(k0) + (i) + 1] + w[(i) + 1]); \
    ZKB_SHA_RND(g, h, a, b, c, d, e, f, SHA_K[(k0) + (i) + 2] + w[(i) + 2]); \
    ZKB_SHA_RND(f, g, h, a, b, c, d, e, SHA_K[(k0) + (i) + 3] + w[(i) + 3]); \
    ZKB_SHA_RND(e, f, g, h, a, b, c, d, SHA_K[(k0) + (i) + 4] + w[(i) + 4]); \
    ZKB_SHA_RND(d, e, f, g, h, a, b, c, SHA_K[(k0) + (i) + 5] + w[(i) + 5]); \
    ZKB_SHA_RND(c, d, e, f, g, h, a, b, SHA_K[(k0) + (i) + 6] + w[(i) + 6]); \
    ZKB_SHA_RND(b, c, d, e, f, g, h, a, SHA_K[(k0) + (i) + 7] + w[(i) + 7]);
    ZKB_SHA_RND8(0, 0)
    ZKB_SHA_RND8(0, 8)
    // Rounds 16..63 as a loop of three 16-round bodies (the schedule window and the renamed working
    // variables both come back to the same registers every 16 rounds): the loop body stays in the
    // instruction cache next to whatever else runs on the SM, a fully unrolled compression does not.
#pragma unroll 1
    for (int k0 = 16; k0 < 64; k0 += 16) {
#pragma unroll
        for (int j = 0; j < 8; j++) ZKB_SHA_SCHED(j);
        ZKB_SHA_RND8(k0, 0)
#pragma unroll
        for (int j = 8; j < 16; j++) ZKB_SHA_SCHED(j);
        ZKB_SHA_RND8(k0, 8)
    }
#undef ZKB_SHA_RND8
    Sha8 o;
    o.v[0] = hin.v[0] + a; o.v[1] = hin.v[1] + b; o.v[2] = hin.v[2] + c; o.v[3] = hin.v[3] + d;
    o.v[4] = hin.v[4] + e; o.v[5] = hin.v[5] + f; o.v[6] = hin.v[6] + g; o.v[7] = hin.v[7] + h;
    return o;
}

// The 64 rounds alone, with K[t] + W[t] read from shared memory.  The message schedule of a
// block depends only on the block, not on the chaining value, so when many known blocks are
// absorbed in a row the lanes of a warp expand 32 schedules side by side and one lane then runs
// only the (inherently serial) rounds.
//
// A lone warp can issue an instruction every cycle, but the logic and shift pipe takes one every two cycles and the
// multiply pipe another one every two, so additions are moved to the multiply pipe: multiply-adds by a one that the
// compiler cannot see through (it turns a multiply by a literal one back into an add).  Ten of the logic pipe's slots are
// fixed (six rotations, four lop3); of the additions only the three-operand one of a' stays there, in the form
// e' = h + kw + d + ch + s1,  a' = e' + s0 + (maj - d).  With the schedule words read sixteen bytes at a time.
// Measured on B200: a lone lane's 64 rounds, unrolled, 1915 cycles in the form of ZKB_SHA_RND and 1763 in this one (both with words
// read one by one; ZKB_SHA_RND rolled by sixteen 1955); checking 1232 attention rows with the caller's transcript of 15 800 blocks
// 19.2 -> 15.0 ms, 0.87 us a block.  Inside a whole compression, where the schedule's additions compete for the same pipes, this
// form is slower than ZKB_SHA_RND.
// Unrolled over the block.  The same rolled by sixteen rounds, rolled -> unrolled: that check 15.9 -> 15.0 ms, the GPT-2 shape 53.1 ->
// 52.6, four 4B-shape layers no difference, thirty-two side by side on one GPU 25.0 -> 25.6 (25.9 before this form).
constexpr int SHA_KW_STRIDE = 68;    // whole 16-byte vectors; lanes that write their own row stay on different banks
__constant__ u32 SHA_ONE = 1u;
__device__ __forceinline__ u32 sha_madd(u32 a, u32 one, u32 b) { u32 r; asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(one), "r"(b)); return r; }
#define ZKB_SHA_RND_KW(a, b, c, d, e, f, g, h, kw)                                 \
    {                                                                             \
        const u32 ch_ = sha_ch(e, f, g);                                          \
        const u32 mj_ = sha_maj(a, b, c);                                         \
        const u32 s1_ = sha_xor3(rotr32(e, 6), rotr32(e, 11), rotr32(e, 25));     \
        const u32 s0_ = sha_xor3(rotr32(a, 2), rotr32(a, 13), rotr32(a, 22));     \
        const u32 y_ = sha_madd(sha_madd(h, one, (kw)), one, d);                  \
        const u32 md_ = sha_madd(d, minus_one, mj_);                              \
        d = sha_madd(sha_madd(y_, one, ch_), one, s1_);                           \
        h = d + s0_ + md_;                                                        \
    }
// kw is shared memory that other lanes have just written and will write again: the loads below say that they read it ("memory"),
// so no store is moved across them whatever the call is inlined into.
__device__ __noinline__ Sha8 sha256_rounds(Sha8 hin, const u32* kw) {
    u32 one = SHA_ONE, minus_one = 0u - SHA_ONE;
    asm volatile("" : "+r"(one), "+r"(minus_one));
    const u32 kwa = (u32)__cvta_generic_to_shared(kw);
    u32 a = hin.v[0], b = hin.v[1], c = hin.v[2], d = hin.v[3], e = hin.v[4], f = hin.v[5], g = hin.v[6], h = hin.v[7];
#pragma unroll
    for (int i = 0; i < 64; i += 8) {
        u32 k[8];
#pragma unroll
        for (int j = 0; j < 8; j += 4)
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(k[j]), "=r"(k[j + 1]), "=r"(k[j + 2]), "=r"(k[j + 3]) : "r"(kwa + 4 * (i + j)) : "memory");
        ZKB_SHA_RND_KW(a, b, c, d, e, f, g, h, k[0]);
        ZKB_SHA_RND_KW(h, a, b, c, d, e, f, g, k[1]);
        ZKB_SHA_RND_KW(g, h, a, b, c, d, e, f, k[2]);
        ZKB_SHA_RND_KW(f, g, h, a, b, c, d, e, k[3]);
        ZKB_SHA_RND_KW(e, f, g, h, a, b, c, d, k[4]);
        ZKB_SHA_RND_KW(d, e, f, g, h, a, b, c, k[5]);
        ZKB_SHA_RND_KW(c, d, e, f, g, h, a, b, k[6]);
        ZKB_SHA_RND_KW(b, c, d, e, f, g, h, a, k[7]);
    }
    Sha8 o;
    o.v[0] = hin.v[0] + a; o.v[1] = hin.v[1] + b; o.v[2] = hin.v[2] + c; o.v[3] = hin.v[3] + d;
    o.v[4] = hin.v[4] + e; o.v[5] = hin.v[5] + f; o.v[6] = hin.v[6] + g; o.v[7] = hin.v[7] + h;
    return o;
}
// Lane-local: expand the schedule of one block (16 big-endian words) into K + W (16-byte aligned).  A loop of sixteen words: it runs
// beside the rounds of the batch before it, whose instruction fetches it must not crowd out.
__device__ __forceinline__ void sha256_expand_kw(const u32* __restrict__ blk_be, u32* kw) {
    u32 w[16];
#pragma unroll
    for (int i = 0; i < 16; i++) w[i] = blk_be[i];
#pragma unroll 1
    for (int i = 0; i < 64; i += 16) {
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            u32 k[4];
#pragma unroll
            for (int z = 0; z < 4; z++) {
                if (i) ZKB_SHA_SCHED(j + z);
                k[z] = SHA_K[i + j + z] + w[j + z];
            }
            *reinterpret_cast<uint4*>(kw + i + j) = make_uint4(k[0], k[1], k[2], k[3]);
        }
    }
}

// Working copy used by the thread (Tr) or the warp (TrWarp, TrPair, below) that advances the transcript.  `buf` points to
// TR_SCRATCH_BYTES of 16-byte-aligned shared memory: the 64-byte message block, then what a pair of warps shares: the 64
// words K + W of the block being compressed, a digest that is the message, and the order to the second warp.
constexpr int TR_SCRATCH_BYTES = 64 + 64 * 4 + 64;

struct Tr {
    u32 h[8];
    u32 buflen;
    u64 total;
    unsigned char* buf;
};

// ---- a compression shared by two warps ------------------------------------------------------------
// More than a third of a fused compression's time is the message schedule, which does not depend on the chaining
// value.  Where a CTA has a warp to spare, that warp (on another scheduler) expands it: the hashing warp writes the
// message, arrives at a named barrier and runs rounds 0..15, for which it has the words; meanwhile the second warp
// expands W[16..31] + K and hands them over through a second barrier, then the other 32 through a third.  A schedule
// word takes it less than a round, so it stays ahead from there on.  The hashing warp runs its code with all lanes in step
// (they hold the same state), so that the barriers see whole warps.
// What bounds it is 64 dependent rounds at 27 cycles, and the size of the code: next to the table work of a tail or to
// other streams' kernels, loops of sixteen rounds for the one warp and of sixteen words for the other are faster than
// unrolled ones.  Measured on B200, whole calls in us (before, fused in one thread / both warps unrolled / both in loops): four 4B-shape
// layers 17690 / 19400 / 16200, their verifier 16450 / 16870 / 14920, the 1024-2048-1024-10 MLP 1522 / 1525 / 1352, a sumcheck
// of 2^12 elements 237 / 225 / 211.
struct TrWarp : Tr {};           // all lanes of a warp in step, compressing alone
struct TrPair : TrWarp {};       // with the second warp
constexpr u32 TRP_KW = 64, TRP_MSG = TRP_KW + 64 * 4, TRP_ORDER = TRP_MSG + 8 * 4;      // byte offsets behind `buf`
static_assert(TRP_ORDER + 4 <= TR_SCRATCH_BYTES, "scratch of a pair");
enum : u32 { TRP_STOP = 0, TRP_BLOCK = 1, TRP_DIGEST = 2 };        // orders: leave; expand the block in `buf`; expand a digest || its padding
constexpr int TRP_BAR_ORDER = 2, TRP_BAR_FIRST = 3, TRP_BAR_REST = 4;    // named barriers (0: the CTA, 1: workers of the pipelined tail)
template <int B> __device__ __forceinline__ void trp_arrive() { asm volatile("bar.arrive %0, 64;" ::"n"(B) : "memory"); }
template <int B> __device__ __forceinline__ void trp_sync() { asm volatile("bar.sync %0, 64;" ::"n"(B) : "memory"); }
__device__ __forceinline__ u32 sh_addr(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sh_ld4(u32 a, u32* o) { asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3]) : "r"(a) : "memory"); }
__device__ __forceinline__ void sh_st4(u32 a, const u32* v) { asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory"); }
__device__ __forceinline__ u32 sh_ld(u32 a) { u32 v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory"); return v; }
__device__ __forceinline__ void sh_st(u32 a, u32 v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
#define ZKB_SHA_RND8_KW(k)                                                                                                                    \
    ZKB_SHA_RND_KW(a, b, c, d, e, f, g, h, (k)[0]); ZKB_SHA_RND_KW(h, a, b, c, d, e, f, g, (k)[1]); ZKB_SHA_RND_KW(g, h, a, b, c, d, e, f, (k)[2]); \
    ZKB_SHA_RND_KW(f, g, h, a, b, c, d, e, (k)[3]); ZKB_SHA_RND_KW(e, f, g, h, a, b, c, d, (k)[4]); ZKB_SHA_RND_KW(d, e, f, g, h, a, b, c, (k)[5]); \
    ZKB_SHA_RND_KW(c, d, e, f, g, h, a, b, (k)[6]); ZKB_SHA_RND_KW(b, c, d, e, f, g, h, a, (k)[7]);
// The hashing warp's rounds, all lanes; kw[0..15] are its own.
__device__ __noinline__ Sha8 sha256_rounds_pair(Sha8 hin, const unsigned char* buf) {
    u32 one = SHA_ONE, minus_one = 0u - SHA_ONE;
    asm volatile("" : "+r"(one), "+r"(minus_one));
    const u32 kw = sh_addr(buf) + TRP_KW;
    u32 a = hin.v[0], b = hin.v[1], c = hin.v[2], d = hin.v[3], e = hin.v[4], f = hin.v[5], g = hin.v[6], h = hin.v[7];
#pragma unroll 1
    for (u32 i = 0; i < 4; i++) {
        if (i == 1) trp_sync<TRP_BAR_FIRST>();
        if (i == 2) trp_sync<TRP_BAR_REST>();
        u32 k[16];
#pragma unroll
        for (int j = 0; j < 16; j += 4) sh_ld4(kw + 64 * i + 4 * j, k + j);
        ZKB_SHA_RND8_KW(k)
        ZKB_SHA_RND8_KW(k + 8)
    }
    __syncwarp();
    Sha8 o;
    o.v[0] = hin.v[0] + a; o.v[1] = hin.v[1] + b; o.v[2] = hin.v[2] + c; o.v[3] = hin.v[3] + d;
    o.v[4] = hin.v[4] + e; o.v[5] = hin.v[5] + f; o.v[6] = hin.v[6] + g; o.v[7] = hin.v[7] + h;
    return o;
}
// The block in `buf` (16 little-endian words).
__device__ __forceinline__ Sha8 sha256_compress_pair(Sha8 hin, const unsigned char* buf) {
    const u32 sb = sh_addr(buf);
    sh_st(sb + TRP_ORDER, TRP_BLOCK);
    __syncwarp();
    trp_arrive<TRP_BAR_ORDER>();
    u32 k[16];
#pragma unroll
    for (int i = 0; i < 16; i += 4) sh_ld4(sb + 4 * i, k + i);
#pragma unroll
    for (int i = 0; i < 16; i++) k[i] = SHA_K[i] + bswap32(k[i]);
#pragma unroll
    for (int i = 0; i < 16; i += 4) sh_st4(sb + TRP_KW + 4 * i, k + i);
    return sha256_rounds_pair(hin, buf);
}
// A digest as the whole message, from the initial state.
__device__ __forceinline__ Sha8 sha256_digest_pair(const Sha8& m, const unsigned char* buf) {
    const u32 sb = sh_addr(buf);
    sh_st4(sb + TRP_MSG, m.v); sh_st4(sb + TRP_MSG + 16, m.v + 4);
    sh_st(sb + TRP_ORDER, TRP_DIGEST);
    __syncwarp();
    trp_arrive<TRP_BAR_ORDER>();
    u32 k[16];
#pragma unroll
    for (int i = 0; i < 16; i++) k[i] = SHA_K[i] + (i < 8 ? m.v[i & 7] : (i == 8 ? 0x80000000u : (i == 15 ? 256u : 0u)));
#pragma unroll
    for (int i = 0; i < 16; i += 4) sh_st4(sb + TRP_KW + 4 * i, k + i);
    return sha256_rounds_pair(Sha8{{0x6a09e667u, 0xbb67ae85u, 0x3c6ef372u, 0xa54ff53au, 0x510e527fu, 0x9b05688cu, 0x1f83d9abu, 0x5be0cd19u}}, buf);
}
// The hashing warp's part in a kernel that does nothing else (chains, verifiers): one loop of eight rounds, the first sixteen words
// straight from the block.  There it is the faster form, in the tails the one above is.  Measured on B200 (that one -> this one):
// checking four 4B-shape layers 14.90 -> 13.95 ms, Basefold of 2^24 coefficients 2886 -> 2785 us, a batch of seven 2300 -> 2208 us; with
// this one in the tails too, four layers proved 16.08 -> 16.30 ms, the GPT-2 shape 47.2 -> 48.6 ms.
struct TrChain : TrPair {};
__device__ __noinline__ Sha8 sha256_compress_chain(Sha8 hin, const unsigned char* buf) {
    u32 one = SHA_ONE, minus_one = 0u - SHA_ONE;
    asm volatile("" : "+r"(one), "+r"(minus_one));
    const u32 sb = sh_addr(buf), kw = sb + TRP_KW;
    sh_st(sb + TRP_ORDER, TRP_BLOCK);
    __syncwarp();
    trp_arrive<TRP_BAR_ORDER>();
    u32 k[16];
#pragma unroll
    for (int i = 0; i < 16; i += 4) sh_ld4(sb + 4 * i, k + i);
#pragma unroll
    for (int i = 0; i < 16; i++) k[i] = SHA_K[i] + bswap32(k[i]);
    u32 a = hin.v[0], b = hin.v[1], c = hin.v[2], d = hin.v[3], e = hin.v[4], f = hin.v[5], g = hin.v[6], h = hin.v[7];
#pragma unroll 1
    for (u32 i = 0;; i++) {
        ZKB_SHA_RND8_KW(k)
        if (i == 7) break;
        if (i & 1) {
            if (i == 1) trp_sync<TRP_BAR_FIRST>();
            if (i == 3) trp_sync<TRP_BAR_REST>();
#pragma unroll
            for (int j = 0; j < 16; j += 4) sh_ld4(kw + 32 * (i + 1) + 4 * j, k + j);
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) k[j] = k[8 + j];
        }
    }
    __syncwarp();
    Sha8 o;
    o.v[0] = hin.v[0] + a; o.v[1] = hin.v[1] + b; o.v[2] = hin.v[2] + c; o.v[3] = hin.v[3] + d;
    o.v[4] = hin.v[4] + e; o.v[5] = hin.v[5] + f; o.v[6] = hin.v[6] + g; o.v[7] = hin.v[7] + h;
    return o;
}
// The second warp's part, all lanes: serves compressions until tr_pair_end.  A kernel that uses a pair is launched with two whole
// warps at least (the chains and the verifiers' kernels with exactly 64 threads), both of which reach their part: the hand-overs
// are barriers of 64 threads, at which a lone warp would wait for good.
//  Two words a step: even lanes the even schedule
// words, odd lanes the odd ones.  With x[j] = W[2j + l] and z[j] = W[2j - 1 + l] (words of the other lane) a step is
// x[j] = sig1(x[j-1]) + z[j-3] + sig0(z[j-7]) + x[j-8].
__device__ __forceinline__ u32 sha_sig0(u32 v) { return sha_xor3(rotr32(v, 7), rotr32(v, 18), v >> 3); }
__device__ __forceinline__ u32 sha_sig1(u32 v) { return sha_xor3(rotr32(v, 17), rotr32(v, 19), v >> 10); }
__device__ __noinline__ void tr_pair_help(const unsigned char* buf) {
    const u32 sb = sh_addr(buf), l = threadIdx.x & 1;
    for (;;) {
        __syncwarp();
        trp_sync<TRP_BAR_ORDER>();
        const u32 order = sh_ld(sb + TRP_ORDER);
        if (order == TRP_STOP) return;
        u32 x[8], z[8];
        z[0] = 0;
        if (order == TRP_DIGEST) {
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] = sh_ld(sb + TRP_MSG + 8 * j + 4 * l);
#pragma unroll
            for (int j = 1; j < 4; j++) z[j] = sh_ld(sb + TRP_MSG + 8 * j - 4 + 4 * l);
            z[4] = sh_ld(sb + TRP_MSG + 28);
            if (l) z[4] = 0x80000000u;
            x[4] = l ? 0u : 0x80000000u; x[5] = x[6] = 0; x[7] = l ? 256u : 0u;
            z[5] = z[6] = z[7] = 0;
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = bswap32(sh_ld(sb + 8 * j + 4 * l));
#pragma unroll
            for (int j = 1; j < 8; j++) z[j] = bswap32(sh_ld(sb + 8 * j - 4 + 4 * l));
        }
#pragma unroll 1
        for (u32 i = 0; i < 3; i++) {
            u32 kk[8];
#pragma unroll
            for (int j = 0; j < 8; j++) kk[j] = SHA_K[16 + 16 * i + 2 * j + l];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const u32 v = sha_sig1(x[(j + 7) & 7]) + (z[(j + 5) & 7] + (sha_sig0(z[(j + 1) & 7]) + x[j]));
                sh_st(sb + TRP_KW + 64 + 64 * i + 8 * j + 4 * l, v + kk[j]);
                z[j] = __shfl_xor_sync(0xffffffffu, l ? x[(j + 7) & 7] : v, 1);
                x[j] = v;
            }
            if (i == 0) trp_arrive<TRP_BAR_FIRST>();
        }
        trp_arrive<TRP_BAR_REST>();
    }
}
// The hashing warp compresses with TrPair only while exactly one other warp of the CTA is in tr_pair_help; this sends it out.  A CTA
// barrier lies between that and the next such stretch (the second warp still reads the order).
__device__ __forceinline__ void tr_pair_end(const TrPair& t) {
    sh_st(sh_addr(t.buf) + TRP_ORDER, TRP_STOP);
    __syncwarp();
    trp_arrive<TRP_BAR_ORDER>();
}

__device__ __forceinline__ void tr_iv(u32 h[8]) {
    h[0] = 0x6a09e667u; h[1] = 0xbb67ae85u; h[2] = 0x3c6ef372u; h[3] = 0xa54ff53au;
    h[4] = 0x510e527fu; h[5] = 0x9b05688cu; h[6] = 0x1f83d9abu; h[7] = 0x5be0cd19u;
}
template <class T>
__device__ __forceinline__ void tr_load(T& t, const TrState* g, unsigned char* scratch) {
#pragma unroll
    for (int i = 0; i < 8; i++) t.h[i] = g->h[i];
    t.buflen = g->buflen;
    t.total = g->total;
    t.buf = scratch;
    const u32* src = reinterpret_cast<const u32*>(g->buf);
    u32* dst = reinterpret_cast<u32*>(scratch);
#pragma unroll
    for (int i = 0; i < 16; i++) dst[i] = src[i];
}
__device__ __forceinline__ void tr_store(const Tr& t, TrState* g) {
#pragma unroll
    for (int i = 0; i < 8; i++) g->h[i] = t.h[i];
    g->buflen = t.buflen;
    g->total = t.total;
    u32* dst = reinterpret_cast<u32*>(g->buf);
    const u32* src = reinterpret_cast<const u32*>(t.buf);
#pragma unroll
    for (int i = 0; i < 16; i++) dst[i] = src[i];
}
__device__ __forceinline__ void tr_flush_block(Tr& t) {
    Sha8 h;
#pragma unroll
    for (int i = 0; i < 8; i++) h.v[i] = t.h[i];
    // Measured on B200 (one thread, ~11 cycles between dependent instructions): the fused
    // schedule + rounds below takes ~3030 cycles, expanding first and then running the rounds ~3830.
    h = sha256_compress(h, reinterpret_cast<const u32*>(t.buf));
#pragma unroll
    for (int i = 0; i < 8; i++) t.h[i] = h.v[i];
    t.buflen = 0;
}
__device__ __forceinline__ void tr_flush_block(TrWarp& t) {
    __syncwarp();
    tr_flush_block(static_cast<Tr&>(t));
    __syncwarp();
}
__device__ __forceinline__ void tr_flush_block(TrPair& t) {
    Sha8 h;
#pragma unroll
    for (int i = 0; i < 8; i++) h.v[i] = t.h[i];
    h = sha256_compress_pair(h, t.buf);
#pragma unroll
    for (int i = 0; i < 8; i++) t.h[i] = h.v[i];
    t.buflen = 0;
}
__device__ __forceinline__ void tr_flush_block(TrChain& t) {
    Sha8 h;
#pragma unroll
    for (int i = 0; i < 8; i++) h.v[i] = t.h[i];
    h = sha256_compress_chain(h, t.buf);
#pragma unroll
    for (int i = 0; i < 8; i++) t.h[i] = h.v[i];
    t.buflen = 0;
}
template <class T>
__device__ __forceinline__ void tr_absorb_byte(T& t, unsigned char c) {
    t.buf[t.buflen++] = c;
    t.total++;
    if (t.buflen == 64) tr_flush_block(t);
}
template <class T>
__device__ __forceinline__ void tr_absorb_u32(T& t, u32 v) {
    if ((t.buflen & 3) == 0) {           // aligned fast path: one word store
        *reinterpret_cast<u32*>(t.buf + t.buflen) = v;
        t.buflen += 4;
        t.total += 4;
        if (t.buflen == 64) tr_flush_block(t);
    } else {
        tr_absorb_byte(t, (unsigned char)v);
        tr_absorb_byte(t, (unsigned char)(v >> 8));
        tr_absorb_byte(t, (unsigned char)(v >> 16));
        tr_absorb_byte(t, (unsigned char)(v >> 24));
    }
}
// N words at once; when the stream is word-aligned (the common case) this is N plain stores
// plus at most one compression, instead of N rounds of per-byte bookkeeping.
template <int N, class T>
__device__ __forceinline__ void tr_absorb_words(T& t, const u32* w) {
    static_assert(N <= 16, "at most one block boundary inside");
    if ((t.buflen & 3) == 0) {
        u32* bw = reinterpret_cast<u32*>(t.buf);
        const u32 pos = t.buflen >> 2;
        const u32 room = 16 - pos;                     // words that still fit into the open block (1..16)
#pragma unroll
        for (int i = 0; i < N; i++) if ((u32)i < room) bw[pos + i] = w[i];
        if ((u32)N >= room) {
            t.buflen = 64;
            tr_flush_block(t);
#pragma unroll
            for (int i = 0; i < N; i++) if ((u32)i >= room) bw[i - room] = w[i];
            t.buflen = ((u32)N - room) << 2;
        } else {
            t.buflen = (pos + N) << 2;
        }
        t.total += 4 * N;
    } else {
#pragma unroll
        for (int i = 0; i < N; i++) tr_absorb_u32(t, w[i]);
    }
}
template <class T>
__device__ __forceinline__ void tr_absorb_fe(T& t, Fe v) {
    u32 w[4] = {v.x, v.y, v.z, v.w};
    tr_absorb_words<4>(t, w);
}
template <class T>
__device__ inline void tr_absorb_bytes(T& t, const unsigned char* p, u32 n) {
    for (u32 i = 0; i < n; i++) tr_absorb_byte(t, p[i]);
}

// Pad, compress, and restart the stream with the 32-byte digest as its first bytes.  Written
// without loops whose trip count depends on the position: on a lone thread every dependent
// instruction costs about 11 cycles, so the zero fill is fourteen predicated stores, not a counted loop.
template <class T>
__device__ __forceinline__ void tr_finalize_reseed(T& t, u32 digest_be[8]) {
    u64 bits = t.total * 8;
    u32 n = t.buflen;
    u32* bw = reinterpret_cast<u32*>(t.buf);
    if ((n & 3) == 0) {
        bw[n >> 2] = 0x00000080u;                      // 0x80 and three zero bytes
        n += 4;
    } else {
        t.buf[n++] = 0x80;
        while (n & 3) t.buf[n++] = 0;
    }
    u32 first = n >> 2;                                // first word still to be zeroed
    if (n > 56) {
#pragma unroll
        for (u32 i = 14; i < 16; i++) if (i >= first) bw[i] = 0;
        tr_flush_block(t);
        first = 0;
    }
#pragma unroll
    for (u32 i = 0; i < 14; i++) if (i >= first) bw[i] = 0;
    bw[14] = bswap32((u32)(bits >> 32));
    bw[15] = bswap32((u32)bits);
    tr_flush_block(t);
#pragma unroll
    for (int i = 0; i < 8; i++) digest_be[i] = t.h[i];
    tr_iv(t.h);
#pragma unroll
    for (int i = 0; i < 8; i++) bw[i] = bswap32(digest_be[i]);   // digest bytes in stream order
    t.buflen = 32;
    t.total = 32;
}
// The first of a digest's four little-endian 64-bit windows below 2^64 - 4, reduced mod p; false when there is none.
__device__ __forceinline__ bool tr_window(const u32* d, u32& v) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
        u64 raw = (u64)bswap32(d[2 * c]) | ((u64)bswap32(d[2 * c + 1]) << 32);
        if (raw < 0xfffffffffffffffcull) { v = red64(raw); return true; }
    }
    return false;
}
// d: the digest that the stream consists of afterwards.
template <class T>
__device__ __forceinline__ u32 tr_squeeze_digest(T& t, u32* d) {
    u32 v = 0;
    for (int guard = 0; guard < 64; guard++) {        // all four windows rejecting has probability 2^-248
        if (t.buflen == 32 && t.total == 32) {
            // stream == one 32-byte digest (the state right after a squeeze): the padded block is fixed
            u32* bw = reinterpret_cast<u32*>(t.buf);
            bw[8] = 0x00000080u;
#pragma unroll
            for (int i = 9; i < 15; i++) bw[i] = 0;
            bw[15] = 0x00010000u;                     // 256 bits, big-endian
            tr_flush_block(t);
#pragma unroll
            for (int i = 0; i < 8; i++) d[i] = t.h[i];
            tr_iv(t.h);
#pragma unroll
            for (int i = 0; i < 8; i++) bw[i] = bswap32(d[i]);
            t.buflen = 32;
        } else {
            tr_finalize_reseed(t, d);
        }
        if (tr_window(d, v)) break;
    }
    return v;
}
template <class T>
__device__ __forceinline__ u32 tr_squeeze(T& t) { u32 d[8]; return tr_squeeze_digest(t, d); }
// n squeezes in a row, out(i, value) for each.  Behind the first one each message is the digest before it, which the hashing
// warp has in registers.
template <class Out>
__device__ __forceinline__ void tr_squeeze_run(TrPair& t, u32 n, Out out) {
    if (n == 0) return;
    Sha8 d;
    out(0u, tr_squeeze_digest(t, d.v));
    if (n == 1) return;
#pragma unroll 1
    for (u32 i = 1; i < n; i++) {
        u32 v = 0;
        for (int guard = 0; guard < 64; guard++) {
            d = sha256_digest_pair(d, t.buf);
            if (tr_window(d.v, v)) break;
        }
        out(i, v);
    }
    u32* bw = reinterpret_cast<u32*>(t.buf);
#pragma unroll
    for (int i = 0; i < 8; i++) bw[i] = bswap32(d.v[i]);
}
template <class Out>
__device__ __forceinline__ void tr_squeeze_run(TrWarp& t, u32 n, Out out) { for (u32 i = 0; i < n; i++) out(i, tr_squeeze(t)); }
template <class Out>
__device__ __forceinline__ void tr_squeeze_run(TrChain& t, u32 n, Out out) { for (u32 i = 0; i < n; i++) out(i, tr_squeeze(t)); }
template <class T> __device__ __forceinline__ void tr_squeeze_el(T& t, Fp& r) { r.v = tr_squeeze(t); }
template <class T> __device__ __forceinline__ void tr_squeeze_el(T& t, Fe& r) {
    tr_squeeze_run(t, 4, [&](u32 i, u32 v) { if (i == 0) r.x = v; else if (i == 1) r.y = v; else if (i == 2) r.z = v; else r.w = v; });
}

// Warp-cooperative absorb of `total` u32 words produced by load(g), g in [0, total) (any lane may
// call load).  `tr` is meaningful in lane 0 only; tile (512 words) and kw (32 * SHA_KW_STRIDE
// words) are shared-memory scratch.  Must be called by all 32 lanes of one warp.
template <class Load>
__device__ __forceinline__ void tr_absorb_stream_warp_aligned(Tr& tr, u32 total, Load load, u32* bufw, u32 have, u32* tile, u32* kw) {
    const int lane = threadIdx.x & 31;
    u32 pos = 0;
    while (have + (total - pos) >= 16) {
        u32 nb = (have + (total - pos)) / 16;
        if (nb > 32) nb = 32;
        for (u32 j = lane; j < nb * 16; j += 32) tile[j] = bswap32(j < have ? bufw[j] : load(pos + j - have));
        __syncwarp();
        if ((u32)lane < nb) sha256_expand_kw(tile + lane * 16, kw + lane * SHA_KW_STRIDE);
        __syncwarp();
        if (lane == 0) {
            Sha8 h;
#pragma unroll
            for (int i = 0; i < 8; i++) h.v[i] = tr.h[i];
            for (u32 b = 0; b < nb; b++) h = sha256_rounds(h, kw + b * SHA_KW_STRIDE);
#pragma unroll
            for (int i = 0; i < 8; i++) tr.h[i] = h.v[i];
        }
        __syncwarp();
        pos += nb * 16 - have;
        have = 0;
    }
    const u32 rest = total - pos;
    for (u32 j = lane; j < rest; j += 32) bufw[have + j] = load(pos + j);
    __syncwarp();
    if (lane == 0) { tr.buflen = (have + rest) * 4; tr.total += (u64)total * 4; }
}
// A stream that holds 4 * have + s bytes (s = 1..3) takes the words shifted by s bytes: stream word i
// is the funnel shift of data words i - 1 and i, the s pending bytes standing in for word -1, and the
// top s bytes of the last word stay pending.  The blocks are then hashed exactly like aligned ones.
template <class Load>
__device__ __forceinline__ void tr_absorb_stream_warp(Tr& tr, u32 total, Load load, u32* tile, u32* kw) {
    const int lane = threadIdx.x & 31;
    __syncwarp();                      // lane 0's earlier writes to the stream buffer become visible
    const u32 buflen = __shfl_sync(0xffffffffu, tr.buflen, 0);
    u32* bufw = reinterpret_cast<u32*>(__shfl_sync(0xffffffffu, (unsigned long long)tr.buf, 0));
    const u32 s = buflen & 3, have = buflen >> 2;
    if (s == 0) { tr_absorb_stream_warp_aligned(tr, total, load, bufw, have, tile, kw); return; }
    if (total == 0) return;
    const u32 sh = 8 * s;
    const u32 pend = bufw[have] << (32 - sh);
    __syncwarp();
    tr_absorb_stream_warp_aligned(tr, total, [=](u32 g) -> u32 { return __funnelshift_l(g ? load(g - 1) : pend, load(g), sh); },
                                  bufw, have, tile, kw);
    if (lane == 0) {
        bufw[tr.buflen >> 2] = load(total - 1) >> (32 - sh);
        tr.buflen += s;
    }
    __syncwarp();
}

// The same absorb for a CTA of two warps with the loads and the schedule expansion taken off the
// hash chain: while lane 0 of warp 0 runs the rounds of one batch (up to 32 blocks, about 28 us),
// warp 1 fetches the next batch's words and expands its schedules into the other half of the
// double-buffered scratch; the two meet at a CTA barrier per batch.  Called by all 64 threads with
// identical arguments; `tr` is meaningful in warp 0, the same in all its lanes; `bufw` is the stream buffer (shared
// memory) that tr.buf points to; tile holds 2 x 512 words, kw 2 x 32 x SHA_KW_STRIDE, bc 1 word.
template <class T, class Load>
__device__ __forceinline__ void tr_absorb_stream_2w_aligned(T& tr, u32 total, Load load, u32* bufw, u32 have, u32* tile, u32* kw) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto produce = [&](u32 slot, u32 have_, u32 pos, u32 nb) {   // warp 1: words [pos, ...) after `have_` buffered ones
        u32* t = tile + slot * 512;
        u32* k = kw + slot * 32 * SHA_KW_STRIDE;
        for (u32 j = lane; j < nb * 16; j += 32) t[j] = bswap32(j < have_ ? bufw[j] : load(pos + j - have_));
        __syncwarp();
        if ((u32)lane < nb) sha256_expand_kw(t + lane * 16, k + lane * SHA_KW_STRIDE);
    };
    u32 pos = 0;
    u32 nb = (have + total) / 16;
    if (nb > 32) nb = 32;
    if (nb && warp == 1) produce(0, have, 0, nb);
    __syncthreads();
    u32 slot = 0;
    while (nb) {
        const u32 next_pos = pos + nb * 16 - have;
        u32 next_nb = (total - next_pos) / 16;
        if (next_nb > 32) next_nb = 32;
        if (warp == 1) {
            if (next_nb) produce(slot ^ 1, 0, next_pos, next_nb);
        } else {
            const u32* k = kw + slot * 32 * SHA_KW_STRIDE;
            Sha8 h;
#pragma unroll
            for (int i = 0; i < 8; i++) h.v[i] = tr.h[i];
            for (u32 b = 0; b < nb; b++) h = sha256_rounds(h, k + b * SHA_KW_STRIDE);
#pragma unroll
            for (int i = 0; i < 8; i++) tr.h[i] = h.v[i];
        }
        __syncthreads();
        pos = next_pos; have = 0; nb = next_nb; slot ^= 1;
    }
    const u32 rest = total - pos;      // fewer than 16 - have words: they stay in the stream buffer
    if (warp == 0) for (u32 j = lane; j < rest; j += 32) bufw[have + j] = load(pos + j);
    if (warp == 0) { tr.buflen = (have + rest) * 4; tr.total += (u64)total * 4; }
    __syncthreads();
}
template <class T, class Load>
__device__ __forceinline__ void tr_absorb_stream_2w(T& tr, u32 total, Load load, u32* bufw, u32* tile, u32* kw, u32* bc) {
    if (threadIdx.x == 0) bc[0] = tr.buflen;
    __syncthreads();                   // also: thread 0's earlier writes to the stream buffer become visible
    const u32 buflen = bc[0];
    const u32 s = buflen & 3, have = buflen >> 2;
    if (s == 0) { tr_absorb_stream_2w_aligned(tr, total, load, bufw, have, tile, kw); return; }
    if (total == 0) { __syncthreads(); return; }
    // byte-misaligned stream (a label of odd length in front, for instance): the same pipeline over funnel-shifted words
    const u32 sh = 8 * s;
    const u32 pend = bufw[have] << (32 - sh);
    __syncthreads();                   // every thread holds the pending bytes before the buffer is written again
    tr_absorb_stream_2w_aligned(tr, total, [=](u32 g) -> u32 { return __funnelshift_l(g ? load(g - 1) : pend, load(g), sh); },
                                bufw, have, tile, kw);
    if (threadIdx.x < 32) {
        bufw[tr.buflen >> 2] = load(total - 1) >> (32 - sh);
        tr.buflen += s;
    }
    __syncthreads();
}

}  // namespace zkb
