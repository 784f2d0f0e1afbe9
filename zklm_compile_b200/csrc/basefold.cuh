// Basefold polynomial commitment, single polynomial
// (rust/zk_ml_prover/src/proving/basefold.rs:106-585).
//
//   tables      T = 1 + (u32 LE of the blake3 XOF of a per-size seed) mod (p - 1), 2^L - 1 values,
//               level i (2^i values) at offset 2^i - 1; w = 1 / (2 T)               basefold.rs:106-157, 323-328
//   encode      cw = [c || c]; level l: chunks of 2^(l+1), L' = L + T R, R' = L - T R   basefold.rs:169-238
//   fold        cw'[j] = (l + r) / 2 + alpha (l - r) w[j mod |w|], l = cw[j], r = cw[j + half]   basefold.rs:250-316
//   opening     per round: alpha, fold coefficients and codeword, Merkle tree of the folded
//               codeword, absorb root, 24 query positions, openings in both trees    basefold.rs:483-585
//
// Encoding never mixes the two halves of [c || c] (chunks are at most 2^log_n long), so a codeword is two equal
// halves, and so are the leaves of its tree: an opening stores one half (v), builds the tree over v and one node over
// (root, root), and takes paths from the half tree.  The first fold has l = r everywhere, so it returns v whatever the
// challenge is: v and its tree are the folded codeword and its tree (only the coefficients are folded for the final
// value), unless a batch adds another codeword to it.  At 2^24 coefficients this leaves 2^25 node hashes of 2^26.
//
// XOF output block b of a root node is one compression with counter b, so the tables are
// generated one 64-byte block per thread.  Encoding levels below
// 2^12 run in shared memory in one pass; higher levels go six at a time through tiles of
// 64 consecutive values x 64 strided rows.  Each fold is fused with the first ten levels of the
// Merkle tree over its output.  The whole opening runs without host round trips: challenges,
// roots, query positions and the raw authentication paths are written to the proof record.
#pragma once
#include "engine.cuh"
#include "merkle.cuh"
#include <algorithm>
#include <map>
#include <mutex>

namespace zkb {

// Full 16-word output of the blake3 compression (needed for XOF blocks).
__device__ inline void b3_compress16(const u32* cv, const u32* m, u32 counter_lo, u32 counter_hi, u32 blen, u32 flags, u32* out16) {
    u32 s0 = cv[0], s1 = cv[1], s2 = cv[2], s3 = cv[3], s4 = cv[4], s5 = cv[5], s6 = cv[6], s7 = cv[7];
    u32 s8 = 0x6a09e667u, s9 = 0xbb67ae85u, s10 = 0x3c6ef372u, s11 = 0xa54ff53au;
    u32 s12 = counter_lo, s13 = counter_hi, s14 = blen, s15 = flags;
    u32 w[16];
#pragma unroll
    for (int i = 0; i < 16; i++) w[i] = m[i];
#pragma unroll
    for (int r = 0; r < 7; r++) {
        B3_G(s0, s4, s8, s12, w[0], w[1]);   B3_G(s1, s5, s9, s13, w[2], w[3]);
        B3_G(s2, s6, s10, s14, w[4], w[5]);  B3_G(s3, s7, s11, s15, w[6], w[7]);
        B3_G(s0, s5, s10, s15, w[8], w[9]);  B3_G(s1, s6, s11, s12, w[10], w[11]);
        B3_G(s2, s7, s8, s13, w[12], w[13]); B3_G(s3, s4, s9, s14, w[14], w[15]);
        if (r < 6) {
            u32 t[16] = {w[2], w[6], w[3], w[10], w[7], w[0], w[4], w[13], w[1], w[11], w[12], w[5], w[9], w[14], w[15], w[8]};
#pragma unroll
            for (int i = 0; i < 16; i++) w[i] = t[i];
        }
    }
    out16[0] = s0 ^ s8;   out16[1] = s1 ^ s9;   out16[2] = s2 ^ s10;  out16[3] = s3 ^ s11;
    out16[4] = s4 ^ s12;  out16[5] = s5 ^ s13;  out16[6] = s6 ^ s14;  out16[7] = s7 ^ s15;
    out16[8] = s8 ^ cv[0];   out16[9] = s9 ^ cv[1];   out16[10] = s10 ^ cv[2];  out16[11] = s11 ^ cv[3];
    out16[12] = s12 ^ cv[4]; out16[13] = s13 ^ cv[5]; out16[14] = s14 ^ cv[6];  out16[15] = s15 ^ cv[7];
}

struct BfSeed { u32 w[8]; };

// One thread = one XOF block = 16 table entries and their fold weights (one inversion per thread).
__global__ void __launch_bounds__(128) bf_tables_kernel(BfSeed seed, size_t total, u32* __restrict__ t_flat, u32* __restrict__ w_flat) {
    const size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b * 16 >= total) return;
    u32 cv[8], m[16], o[16];
#pragma unroll
    for (int i = 0; i < 8; i++) { cv[i] = B3_IV[i]; m[i] = seed.w[i]; m[8 + i] = 0; }
    b3_compress16(cv, m, (u32)b, (u32)(b >> 32), 32, B3_CHUNK_START | B3_CHUNK_END | B3_ROOT, o);
    u32 t[16], pre[16];
    u32 acc = 1;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        t[i] = 1 + o[i] % (ZKB_P - 1);
        pre[i] = acc;
        acc = mul31(acc, add31(t[i], t[i]));
    }
    u32 inv = inv31(acc);
#pragma unroll
    for (int i = 15; i >= 0; i--) {
        u32 wv = mul31(pre[i], inv);
        inv = mul31(inv, add31(t[i], t[i]));
        size_t g = b * 16 + i;
        if (g < total) { t_flat[g] = t[i]; w_flat[g] = wv; }
    }
}

// ---- encode -------------------------------------------------------------------------------------
struct CoefSrc { const u32* p; u32 rows, cols, log_cols_pad; };

constexpr int BF_LOW_LOG = 12;
// Levels 0..K-1 of a polynomial of 2^K coefficients (K < BF_LOW_LOG): one CTA, entirely in shared memory.
__global__ void __launch_bounds__(256) bf_encode_low_kernel(CoefSrc src, u32 K, const u32* __restrict__ t_flat, u32* __restrict__ cw,
                                                            size_t n_pad, int dup) {
    __shared__ u32 s[1 << BF_LOW_LOG];
    __shared__ u32 tw[1 << BF_LOW_LOG];
    const u32 T = 1u << K;
    const size_t base = (size_t)blockIdx.x << K;
    for (u32 i = threadIdx.x; i < T; i += blockDim.x) {
        s[i] = coef_at(src.p, src.rows, src.cols, src.log_cols_pad, base + i);
        if (i + 1 < T) tw[i] = t_flat[i];
    }
    __syncthreads();
    for (u32 l = 0; l < K; l++) {
        const u32 half = 1u << l;
        for (u32 b = threadIdx.x; b < T / 2; b += blockDim.x) {
            u32 j = b & (half - 1);
            u32 iL = ((b >> l) << (l + 1)) + j, iR = iL + half;
            u32 rhs = mul31(s[iR], tw[half - 1 + j]);
            u32 L = s[iL];
            s[iL] = add31(L, rhs);
            s[iR] = sub31(L, rhs);
        }
        __syncthreads();
    }
    for (u32 i = threadIdx.x; i < T; i += blockDim.x) {
        cw[base + i] = s[i];
        if (dup) cw[n_pad + base + i] = s[i];
    }
}
// A butterfly level over 2^NS values of a thread; tw[2^s - 1 + j] is the factor of level s for position j of a half.
template <int NS>
__device__ __forceinline__ void bf_butterflies(u32* e, const u32* tw) {
#pragma unroll
    for (int s = 0; s < NS; s++) {
#pragma unroll
        for (int k = 0; k < (1 << NS); k++) {
            if (k & (1 << s)) continue;
            const u32 r = mul31(e[k | (1 << s)], tw[(1 << s) - 1 + (k & ((1 << s) - 1))]), l = e[k];
            e[k] = add31(l, r);
            e[k | (1 << s)] = sub31(l, r);
        }
    }
}
// Levels 0..11 on tiles of 2^12 coefficients, four levels at a time on sixteen values in a thread's registers: three trips
// through shared memory instead of twelve, and fifteen factors for 32 butterflies.  One word of padding per sixteen keeps
// the strided accesses on different banks.
// Bound by integer issue behind the loads of coefficients and factors (ncu at 2^22: ALU pipe 55 %, shared memory 17 %, DRAM 6 %).  Measured
// on B200 with a level at a time in shared memory -> with this and the high levels three at a time: a whole opening of 2^24
// coefficients 3053 -> 2929 us, encoding both halves of them 389 -> 259 us.
__global__ void __launch_bounds__(256) bf_encode_low12_kernel(CoefSrc src, const u32* __restrict__ t_flat, u32* __restrict__ cw, size_t n_pad, int dup) {
    __shared__ u32 sm[(1 << BF_LOW_LOG) + (1 << (BF_LOW_LOG - 4))];
    const size_t base = (size_t)blockIdx.x << BF_LOW_LOG;
    const u32 t = threadIdx.x;
    for (u32 i = t; i < (1u << BF_LOW_LOG); i += 256) sm[i + (i >> 4)] = coef_at(src.p, src.rows, src.cols, src.log_cols_pad, base + i);
    u32 e[16], tw[15];
#pragma unroll
    for (int p = 0; p < 3; p++) {
        const u32 lo = t & ((1u << (4 * p)) - 1), first = ((t >> (4 * p)) << (4 * p + 4)) | lo;
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
            for (int j = 0; j < (1 << s); j++) tw[(1 << s) - 1 + j] = t_flat[(1u << (4 * p + s)) - 1 + ((u32)j << (4 * p)) + lo];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k++) { const u32 i = first + ((u32)k << (4 * p)); e[k] = sm[i + (i >> 4)]; }
        bf_butterflies<4>(e, tw);
        if (p < 2) {                                   // the same thread wrote what it read: no barrier in between
#pragma unroll
            for (int k = 0; k < 16; k++) { const u32 i = first + ((u32)k << (4 * p)); sm[i + (i >> 4)] = e[k]; }
        }
    }
#pragma unroll
    for (int k = 0; k < 16; k++) {
        cw[base + t + 256 * k] = e[k];
        if (dup) cw[n_pad + base + t + 256 * k] = e[k];
    }
}
// Stages s0 .. s0 + NS - 1 of a high tile (rows of 64 values, row stride 2^l0 in the codeword): a thread takes the 2^NS rows
// that these stages combine.  FIRST reads the codeword, LAST writes it; in between the tile is in shared memory.
template <int NS>
__device__ __forceinline__ void bf_high_stages(u32* __restrict__ cw, u32* sm, size_t base, u32 l0, u32 r, u32 s0, const u32* __restrict__ t_flat, size_t col,
                                               bool first, bool last, size_t n_pad, int dup) {
    for (u32 task = threadIdx.x; task < (64u << (r - NS)); task += blockDim.x) {
        const u32 x = task & 63, g = task >> 6;
        const u32 mlow = g & ((1u << s0) - 1), row0 = ((g >> s0) << (s0 + NS)) | mlow;
        u32 e[1 << NS], tw[(1 << NS) - 1];
#pragma unroll
        for (int s = 0; s < NS; s++)
#pragma unroll
            for (int j = 0; j < (1 << s); j++)
                tw[(1 << s) - 1 + j] = t_flat[((size_t(1) << (l0 + s0 + s)) - 1) + ((size_t)(((u32)j << s0) | mlow) << l0) + col + x];
#pragma unroll
        for (int k = 0; k < (1 << NS); k++) {
            const u32 row = row0 + ((u32)k << s0);
            e[k] = first ? cw[base + ((size_t)row << l0) + x] : sm[row * 64 + x];
        }
        bf_butterflies<NS>(e, tw);
#pragma unroll
        for (int k = 0; k < (1 << NS); k++) {
            const u32 row = row0 + ((u32)k << s0);
            if (!last) { sm[row * 64 + x] = e[k]; continue; }
            const size_t at = base + ((size_t)row << l0) + x;
            cw[at] = e[k];
            if (dup) cw[n_pad + at] = e[k];
        }
    }
}
// Levels l0 .. l0+r-1 (r <= 6, l0 >= 6): a CTA holds 2^r rows (stride 2^l0) of 64 consecutive values, up to three levels
// at a time in registers.
__global__ void __launch_bounds__(256) bf_encode_high_kernel(u32* __restrict__ cw, u32 l0, u32 r, const u32* __restrict__ t_flat,
                                                             size_t n_pad, int dup) {
    __shared__ u32 sm[64 * 64];
    const size_t lo_chunks = (size_t(1) << l0) >> 6;
    const size_t H = blockIdx.x / lo_chunks, lc = blockIdx.x % lo_chunks;
    const size_t base = (H << (l0 + r)) + (lc << 6);
    for (u32 s0 = 0; s0 < r;) {
        const u32 left = r - s0, ns = left >= 3 ? 3 : left;
        if (s0) __syncthreads();
        if (ns == 3) bf_high_stages<3>(cw, sm, base, l0, r, s0, t_flat, lc << 6, s0 == 0, left == ns, n_pad, dup);
        else if (ns == 2) bf_high_stages<2>(cw, sm, base, l0, r, s0, t_flat, lc << 6, s0 == 0, left == ns, n_pad, dup);
        else bf_high_stages<1>(cw, sm, base, l0, r, s0, t_flat, lc << 6, s0 == 0, left == ns, n_pad, dup);
        s0 += ns;
    }
}

// ---- per-round transcript step and openings ------------------------------------------------------
constexpr u32 BF_QUERIES = 24;       // pcs.rs:19
struct BfRound {
    // trees: prev has height h_prev over prev_values, folded has height h_prev - 1
    const u32* prev_values; const uint4* prev_nodes;
    const u32* fold_values; const uint4* fold_nodes;
    u32 h_prev;
    int prev_doubled;                // prev_values / prev_nodes hold one half of a codeword [v || v] (height h_prev - 1)
    u32* alpha_next;                 // where the next round's challenge goes (null after the last round)
    u32* rec;                        // [root 4][idx 24][48 prev paths][24 folded paths]
};
// The rounds [first, first + count) of an opening.
constexpr u32 BF_MAX_ROUNDS = 28;
struct BfRounds {
    TrState* tr;
    const u32* point; u32 n_point;   // device-resident evaluation point
    u32 first, count;
    BfRound r[BF_MAX_ROUNDS];
};
__host__ __device__ __forceinline__ size_t bf_round_words(u32 h_prev) {
    size_t pw_prev = 2 + 4 * (size_t)(h_prev - 1), pw_fold = h_prev >= 2 ? 2 + 4 * (size_t)(h_prev - 2) : 2;
    return 4 + BF_QUERIES + 2 * BF_QUERIES * pw_prev + BF_QUERIES * pw_fold;
}
// The challenge of a round: the point coordinate (absorbed) while there is one, else a squeeze
// (basefold.rs:508-513).
template <class T>
__device__ __forceinline__ u32 bf_next_alpha(T& tr, const u32* point, u32 n_point, u32 round) {
    if (round < n_point) { u32 a = point[round]; tr_absorb_u32(tr, a); return a; }
    return tr_squeeze(tr);
}
// The transcript's part of some rounds: absorb the folded root, squeeze the query positions, take the next challenge.  This
// is the opening's critical path (26 dependent SHA-256 compressions a round), so nothing else is in
// it: the paths are gathered by bf_gather_kernel, off the chain.  Measured on B200 with the gathers inside and a launch per
// round -> like this: Basefold of 2^24 coefficients 3213 -> 3053 us.
__global__ void __launch_bounds__(64) bf_chain_kernel(const __grid_constant__ BfRounds a) {
    __shared__ __align__(16) unsigned char trbuf[TR_SCRATCH_BYTES];
    if (threadIdx.x >= 32) { tr_pair_help(trbuf); return; }
    const bool lead = threadIdx.x == 0;
    TrChain tr;
    tr_load(tr, a.tr, trbuf);
    for (u32 round = a.first; round < a.first + a.count; round++) {
        const BfRound& p = a.r[round];
        const u32 h_fold = p.h_prev - 1;
        const uint4 root = p.fold_nodes[mk_layer_offset(h_fold, h_fold)];
        u32 rw[4] = {root.x, root.y, root.z, root.w};
        tr_absorb_words<4>(tr, rw);
        u32* rec = p.rec;
        if (lead) { rec[0] = root.x; rec[1] = root.y; rec[2] = root.z; rec[3] = root.w; }
        const u32 prev_half_mask = (1u << (p.h_prev - 1)) - 1;
        tr_squeeze_run(tr, BF_QUERIES, [=](u32 q, u32 v) { if (lead) rec[4 + q] = v & prev_half_mask; });     // (squeeze mod 2^h_prev) mod prev_half
        if (p.alpha_next) {
            const u32 v = bf_next_alpha(tr, a.point, a.n_point, round + 1);
            if (lead) *p.alpha_next = v;
        }
    }
    tr_pair_end(tr);
    if (lead) tr_store(tr, a.tr);
}
// The opened paths of those rounds, one warp each: blockIdx.y is the round, 3 * BF_QUERIES paths to a round.
constexpr u32 BF_GATHER_WARPS = 8;
__global__ void __launch_bounds__(32 * BF_GATHER_WARPS) bf_gather_kernel(const __grid_constant__ BfRounds a) {
    const BfRound& p = a.r[a.first + blockIdx.y];
    const u32 h_fold = p.h_prev - 1;
    const u32* idx = p.rec + 4;
    const size_t prev_half = size_t(1) << (p.h_prev - 1);
    const size_t pw_prev = 2 + 4 * (size_t)(p.h_prev - 1), pw_fold = h_fold >= 1 ? 2 + 4 * (size_t)(h_fold - 1) : 2;
    u32* out_prev = p.rec + 4 + BF_QUERIES;
    u32* out_fold = out_prev + 2 * BF_QUERIES * pw_prev;
    const u32 lane = threadIdx.x & 31, item = blockIdx.x * BF_GATHER_WARPS + (threadIdx.x >> 5);
    if (item < 2 * BF_QUERIES) {
        const size_t pos = idx[item >> 1] + ((item & 1) ? prev_half : 0);
        if (p.prev_doubled) mk_gather_path_doubled(p.prev_values, p.prev_nodes, h_fold, pos, out_prev + item * pw_prev, lane, 32);
        else mk_gather_path(p.prev_values, size_t(1) << p.h_prev, p.prev_nodes, p.h_prev, pos, out_prev + item * pw_prev, lane, 32);
    } else if (item < 3 * BF_QUERIES) {
        const u32 q = item - 2 * BF_QUERIES;
        mk_gather_path(p.fold_values, prev_half, p.fold_nodes, h_fold, idx[q], out_fold + q * pw_fold, lane, 32);
    }
}
// The first fold of the coefficients (their values at the opened point, one coordinate per round): eval[j] = c[j] + alpha (c[j + half] - c[j]).
// The later ones ride on the codeword folds; the first codeword fold needs no kernel.
__global__ void __launch_bounds__(256) bf_eval_first_kernel(CoefSrc src, const u32* __restrict__ alpha, size_t half, u32* __restrict__ eval) {
    const Fp a{*alpha};
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < half; j += (size_t)gridDim.x * blockDim.x)
        eval[j] = lerp(Fp{coef_at(src.p, src.rows, src.cols, src.log_cols_pad, j)}, Fp{coef_at(src.p, src.rows, src.cols, src.log_cols_pad, j + half)}, a).v;
}
// First challenge, after the commitment root has been absorbed (basefold.rs:461 / 508-513).
__global__ void bf_begin_kernel(TrState* st, const uint4* root, const u32* point, u32 n_point, u32* alpha0, u32* rec_root) {
    __shared__ __align__(16) unsigned char trbuf[TR_SCRATCH_BYTES];
    Tr tr;
    tr_load(tr, st, trbuf);
    uint4 r = *root;
    u32 rw[4] = {r.x, r.y, r.z, r.w};
    tr_absorb_words<4>(tr, rw);
    rec_root[0] = r.x; rec_root[1] = r.y; rec_root[2] = r.z; rec_root[3] = r.w;
    *alpha0 = bf_next_alpha(tr, point, n_point, 0);
    tr_store(tr, st);
}

// ---- host side ----------------------------------------------------------------------------------
struct BfTables { u32* t_flat; u32* w_flat; };

// One table set per (device, log_n) for the life of the process, as the reference caches them
// (basefold.rs:377-393).  The seed is blake3("basefold-foldable-code" || log_n as u64 LE).
inline BfTables bf_tables(zkb_ctx* c, u32 log_n) {
    static std::mutex mu;
    static std::map<std::pair<int, u32>, BfTables> cache;
    std::lock_guard<std::mutex> g(mu);
    auto key = std::make_pair(c->device, log_n);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    const size_t total = (size_t(1) << log_n) - 1;
    BfTables tb{};
    ZKB_CUDA(cudaMalloc(&tb.t_flat, (total + 1) * 4));
    ZKB_CUDA(cudaMalloc(&tb.w_flat, (total + 1) * 4));
    // seed: a 30-byte message hashed on the device through the generic commit path
    u32* seed_dev = (u32*)c->scratch(32);
    unsigned char msg[30];
    memcpy(msg, "basefold-foldable-code", 22);
    for (int i = 0; i < 8; i++) msg[22 + i] = (unsigned char)((uint64_t)log_n >> (8 * i));
    commit_large(c, b3_prefix(msg, 30), nullptr, 0, seed_dev);
    BfSeed seed;
    ZKB_CUDA(cudaMemcpyAsync(seed.w, seed_dev, 32, cudaMemcpyDeviceToHost, c->stream));
    ZKB_CUDA(cudaStreamSynchronize(c->stream));
    const size_t blocks = (total + 15) / 16;
    bf_tables_kernel<<<(unsigned)((blocks + 127) / 128), 128, 0, c->stream>>>(seed, total, tb.t_flat, tb.w_flat);
    ZKB_LAUNCHED(c);
    ZKB_CUDA(cudaStreamSynchronize(c->stream));
    cache[key] = tb;
    return tb;
}

// cw = encode of the zero-padded coefficients: 2^log_n words, the one half of the codeword, or all 2 * 2^log_n words.
inline void bf_encode(zkb_ctx* c, CoefSrc src, u32 log_n, const BfTables& tb, u32* cw, bool both_halves) {
    const size_t n_pad = size_t(1) << log_n;
    const u32 K = log_n < (u32)BF_LOW_LOG ? log_n : (u32)BF_LOW_LOG;
    if (K == (u32)BF_LOW_LOG) bf_encode_low12_kernel<<<(unsigned)(n_pad >> K), 256, 0, c->stream>>>(src, tb.t_flat, cw, n_pad, both_halves && K == log_n);
    else bf_encode_low_kernel<<<(unsigned)(n_pad >> K), 256, 0, c->stream>>>(src, K, tb.t_flat, cw, n_pad, both_halves);
    ZKB_LAUNCHED(c);
    u32 l0 = K;
    while (l0 < log_n) {
        u32 rem = log_n - l0;
        u32 r = rem <= 6 ? rem : (rem < 12 ? (rem + 1) / 2 : 6);
        bf_encode_high_kernel<<<(unsigned)(n_pad >> (r + 6)), 256, 0, c->stream>>>(cw, l0, r, tb.t_flat, n_pad, both_halves && l0 + r == log_n);
        ZKB_LAUNCHED(c);
        l0 += r;
    }
}

template <int KIND>
inline void mk_launch(zkb_ctx* c, int mode, const u32* values, size_t n_valid, size_t n_in, u32 k0, u32 h, uint4* nodes, const MkFold& f) {
    if (n_in >= MK_LANE_MIN) {
        const unsigned grid = (unsigned)(n_in / (MK_LANE_THREADS * MK_LANE));
        if (mode == MK_VALUES) mk_lane_kernel<KIND, MK_VALUES><<<grid, MK_LANE_THREADS, mk_lane_smem(KIND), c->stream>>>(values, n_valid, k0, h, nodes, f);
        else if (mode == MK_DIGESTS) mk_lane_kernel<KIND, MK_DIGESTS><<<grid, MK_LANE_THREADS, mk_lane_smem(KIND), c->stream>>>(values, n_valid, k0, h, nodes, f);
        else mk_lane_kernel<KIND, MK_FOLD><<<grid, MK_LANE_THREADS, mk_lane_smem(KIND), c->stream>>>(values, n_valid, k0, h, nodes, f);
        ZKB_LAUNCHED(c);
        return;
    }
    const size_t tile = n_in < (size_t)MK_TILE ? n_in : (size_t)MK_TILE;
    const unsigned grid = (unsigned)(n_in / tile);
    const bool doubled = f.doubled && grid == 1;
    if (mode == MK_VALUES && doubled) mk_tile_kernel<KIND, MK_VALUES, true><<<grid, MK_THREADS, 0, c->stream>>>(values, n_valid, n_in, k0, h, nodes, f);
    else if (mode == MK_VALUES) mk_tile_kernel<KIND, MK_VALUES, false><<<grid, MK_THREADS, 0, c->stream>>>(values, n_valid, n_in, k0, h, nodes, f);
    else if (mode == MK_DIGESTS && doubled) mk_tile_kernel<KIND, MK_DIGESTS, true><<<grid, MK_THREADS, 0, c->stream>>>(values, n_valid, n_in, k0, h, nodes, f);
    else if (mode == MK_DIGESTS) mk_tile_kernel<KIND, MK_DIGESTS, false><<<grid, MK_THREADS, 0, c->stream>>>(values, n_valid, n_in, k0, h, nodes, f);
    else mk_tile_kernel<KIND, MK_FOLD, false><<<grid, MK_THREADS, 0, c->stream>>>(values, n_valid, n_in, k0, h, nodes, f);
    ZKB_LAUNCHED(c);
}
// Build every layer of a tree of height h; the first launch reads leaves (values, or a fold).
inline void mk_build(zkb_ctx* c, int kind, int first_mode, const u32* values, size_t n_valid, u32 h, uint4* nodes, const MkFold& f) {
    u32 k0 = 0;
    int mode = first_mode;
    while (k0 < h) {
        size_t n_in = size_t(1) << (h - k0);
        if (kind == NODE_AES_MMO) mk_launch<NODE_AES_MMO>(c, mode, values, n_valid, n_in, k0, h, nodes, f);
        else mk_launch<NODE_BLAKE3>(c, mode, values, n_valid, n_in, k0, h, nodes, f);
        const u32 levels = n_in >= MK_LANE_MIN ? (u32)MK_LANE_LOG : (u32)MK_TILE_LOG;
        k0 += (h - k0) < levels ? (h - k0) : levels;
        mode = MK_DIGESTS;
    }
}
inline void aes_tables_upload() {
    static std::mutex mu;
    static std::map<int, bool> done;
    int dev = 0;
    ZKB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    if (done[dev]) return;
    AesTables t = aes_make_tables();
    ZKB_CUDA(cudaMemcpyToSymbol(AES_T0, t.t0, sizeof(t.t0)));
    ZKB_CUDA(cudaMemcpyToSymbol(AES_SBOX, t.sbox, sizeof(t.sbox)));
    // table and staged leaves together exceed the 48 KB that need no opt-in
    ZKB_CUDA(cudaFuncSetAttribute(mk_lane_kernel<NODE_AES_MMO, MK_VALUES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mk_lane_smem(NODE_AES_MMO)));
    ZKB_CUDA(cudaFuncSetAttribute(mk_lane_kernel<NODE_AES_MMO, MK_FOLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mk_lane_smem(NODE_AES_MMO)));
    done[dev] = true;
}

// Record layout of one opening, filled by basefold_enqueue and read by basefold_finish.
struct BfPending {
    u32 log_n = 0;
    size_t num_coeffs = 0;
    size_t root_off = 0, final_off = 0;
    std::vector<size_t> round_off;
};

inline void bf_launch_gather(zkb_ctx* c, const BfRounds& a) {
    bf_gather_kernel<<<dim3((3 * BF_QUERIES + BF_GATHER_WARPS - 1) / BF_GATHER_WARPS, a.count), 32 * BF_GATHER_WARPS, 0, c->stream>>>(a);
    ZKB_LAUNCHED(c);
}
inline void bf_launch_chain(zkb_ctx* c, const BfRounds& a) {
    bf_chain_kernel<<<1, 64, exclusive_smem(bf_chain_kernel, c), c->stream>>>(a);
    ZKB_LAUNCHED(c);
}
// How many rounds the chain launch that starts at `round` takes when the trees run ahead on another stream: one while the
// folded codewords are long (the next tree is still being built when this round's positions are known), then four,
// then all the rest.  With blake3 nodes the line is where a fold and its tree take less than the chain's 30 us a round, so that from there
// on the trees run away from the chain: measured on B200 alone on one stream, blake3 / AES: 2^20 values 71 / 82 us, 2^19 51 / 67, 2^18 37 / 48,
// 2^17 29 / 39, 2^15 27 / 37, 2^10 16 / 24.  AES trees of these sizes stay behind the chain, whose first launch of four rounds then waits for
// them; the line is the same because it measured best there too: 16 below instead of 18 (the line when a round took 46 us), openings of 2^24
// coefficients 2784 -> 2748 us, of 2^20 with AES nodes 1455 -> 1404, a batch of seven with AES nodes 2203 -> 2163; two rounds in the first
// group instead of four: 2820.
inline u32 bf_chain_rounds(u32 round, u32 log_n) {
    const u32 long_rounds = log_n > 16 ? log_n - 16 : 0;
    const u32 n = round < long_rounds ? 1 : (round == long_rounds ? 4 : log_n);
    return n < log_n - round ? n : log_n - round;
}

// One half of a polynomial's codeword and its tree; nothing in it depends on the transcript.
struct BfCommit { u32* cw = nullptr; uint4* tree = nullptr; };
inline void bf_commit_enqueue(zkb_ctx* c, CoefSrc src, u32 log_n, int kind, const BfTables& tb, BfCommit to) {
    c->prof_mark();
    bf_encode(c, src, log_n, tb, to.cw, false);
    c->prof_mark();
    MkFold none{};
    none.doubled = 1;
    mk_build(c, kind, MK_VALUES, to.cw, size_t(1) << log_n, log_n, to.tree, none);
    c->prof_mark();
}

// Enqueue commit + opening of the polynomial `src` (num_coeffs live coefficients, padded view of
// 2^log_n) at the device-resident point.  The transcript first absorbs the commitment root.  `made`: the commitment, if it
// has been made already; what is enqueued on the second stream behind this opening may then use its memory again.
inline BfPending basefold_enqueue(zkb_ctx* c, TrState* tr, CoefSrc src, size_t num_coeffs, u32 log_n, const u32* point_dev, u32 n_point,
                                  int kind, const BfCommit* made = nullptr) {
    if (log_n < 1 || log_n > 28) throw ArgFail{ZKB_E_TOO_LARGE, "basefold: log_n out of range"};
    if (kind != NODE_BLAKE3 && kind != NODE_AES_MMO) throw ArgFail{ZKB_E_ARG, "unknown node hash"};
    if (kind == NODE_AES_MMO) aes_tables_upload();
    BfTables tb = bf_tables(c, log_n);
    const size_t n_pad = size_t(1) << log_n;
    BfPending pd;
    pd.log_n = log_n; pd.num_coeffs = num_coeffs;
    // Every fold challenge that is a coordinate of the point is known before the opening starts (it is
    // absorbed, not squeezed: basefold.rs:508-513), so the folds and trees of those rounds do not wait for
    // the transcript: they run ahead on a second stream, each round into buffers of its own, while the
    // context's stream runs the hash chain (root absorb, 24 query squeezes) and the path gathers behind them.
    const bool ahead = n_point >= log_n && !c->opt_bf_in_order;
    u32* cwA = made ? made->cw : (u32*)c->scratch(n_pad * 4);
    u32* cwB = ahead ? nullptr : (u32*)c->scratch(n_pad / 2 * 4);
    u32* eval = (u32*)c->scratch((n_pad / 2 + 4) * 4);
    uint4* treeA = made ? made->tree : (uint4*)c->scratch(mk_node_count(log_n) * 16 + 16);
    uint4* treeB = ahead ? nullptr : (uint4*)c->scratch(mk_node_count(log_n) * 16 + 16);
    u32* alpha = (u32*)c->scratch((log_n + 1) * 4);
    std::vector<u32*> cws{cwA};            // the folded codeword of each round: the first fold's is the codeword's half itself
    std::vector<uint4*> trees{treeA};
    if (ahead) {
        for (u32 round = 1; round < log_n; round++) {
            cws.push_back((u32*)c->scratch((size_t(4) << (log_n - round)) + 16));
            trees.push_back((uint4*)c->scratch(mk_node_count(log_n - round) * 16 + 16));
        }
    }

    if (!made) bf_commit_enqueue(c, src, log_n, kind, tb, BfCommit{cwA, treeA});
    SideFork fork(c, ahead, log_n);
    pd.root_off = c->rec_alloc(4);
    bf_begin_kernel<<<1, 1, 0, c->stream>>>(tr, treeA + mk_node_count(log_n), point_dev, n_point, alpha, c->rec_dev + pd.root_off);
    ZKB_LAUNCHED(c);

    u32* prev_cw = cwA; u32* next_cw = cwA;
    uint4* prev_tree = treeA; uint4* next_tree = treeA;
    BfRounds rounds{};
    rounds.tr = tr; rounds.point = point_dev; rounds.n_point = n_point;
    for (u32 round = 0; round < log_n; round++) {
        const u32 h_prev = log_n + 1 - round;
        const size_t half = size_t(1) << (h_prev - 1);
        const u32 fold_level = log_n - 1 - round;
        MkFold f{};
        f.prev = prev_cw; f.out = next_cw;
        f.weights = tb.w_flat + ((size_t(1) << fold_level) - 1);
        f.w_len = size_t(1) << fold_level;
        f.prev_partner = half;
        f.alpha = ahead ? point_dev + round : alpha + round;
        f.eval_src = eval; f.eval_dst = eval; f.eval_half = half / 2;
        auto fold = [&] {
            if (round == 0) {
                bf_eval_first_kernel<<<grid_for(c, half / 2), 256, 0, c->stream>>>(src, f.alpha, half / 2, eval);
                ZKB_LAUNCHED(c);
            } else mk_build(c, kind, MK_FOLD, nullptr, half, h_prev - 1, next_tree, f);
        };
        c->stream = fork.side;
        fold();
        c->stream = fork.main;
        if (ahead) ZKB_CUDA(cudaEventRecord(c->side_event(round), fork.side));
        c->prof_mark();
        BfRound& rp = rounds.r[round];
        rp.alpha_next = round + 1 < log_n ? alpha + round + 1 : nullptr;
        rp.prev_values = prev_cw; rp.prev_nodes = prev_tree; rp.fold_values = next_cw; rp.fold_nodes = next_tree;
        rp.h_prev = h_prev;
        rp.prev_doubled = round == 0;
        size_t off = c->rec_alloc(bf_round_words(h_prev));
        rp.rec = c->rec_dev + off;
        pd.round_off.push_back(off);
        if (!ahead) {                    // the buffers are used again two rounds later, so the paths are gathered now
            rounds.first = round; rounds.count = 1;
            bf_launch_chain(c, rounds);
            bf_launch_gather(c, rounds);
        }
        c->prof_mark();
        if (ahead) {
            prev_cw = next_cw; prev_tree = next_tree;
            if (round + 1 < log_n) { next_cw = cws[round + 1]; next_tree = trees[round + 1]; }
        } else if (round == 0) {
            next_cw = cwB; next_tree = treeB;
        } else {
            std::swap(prev_cw, next_cw);
            std::swap(prev_tree, next_tree);
        }
    }
    if (ahead) {
        // Only rounds 0 and 1 open paths of the commitment.  Where its memory is wanted again they are gathered on the second stream as
        // soon as their positions are known, the others together behind the last round.
        const u32 early = made ? (log_n < 2 ? log_n : 2) : 0;
        bool gathered = early == 0;
        for (u32 first = 0; first < log_n; first += rounds.count) {
            rounds.first = first; rounds.count = bf_chain_rounds(first, log_n);
            ZKB_CUDA(cudaStreamWaitEvent(fork.main, c->side_event(first + rounds.count - 1), 0));
            bf_launch_chain(c, rounds);
            if (!gathered && first + rounds.count >= early) {
                BfRounds r = rounds;
                r.first = 0; r.count = early;
                ZKB_CUDA(cudaEventRecord(c->side_event(log_n + 1), fork.main));
                ZKB_CUDA(cudaStreamWaitEvent(fork.side, c->side_event(log_n + 1), 0));
                c->stream = fork.side;
                bf_launch_gather(c, r);
                c->stream = fork.main;
                gathered = true;
            }
        }
        if (early) fork.join(); else fork.joined();
        rounds.first = early; rounds.count = log_n - early;
        if (rounds.count) bf_launch_gather(c, rounds);
    }
    pd.final_off = c->rec_alloc(1);
    ZKB_CUDA(cudaMemcpyAsync(c->rec_dev + pd.final_off, eval, 4, cudaMemcpyDeviceToDevice, c->stream));
    return pd;
}

// ---- serialisation (host, after the record has been fetched) --------------------------------------
// BatchMerkleProof (pcs.rs:43-53) of `positions` from raw paths: indices and values in caller
// order; per level the digests of the siblings that are not themselves known, ascending
// (pcs.rs:299-330).  raw[i] points at the path record of positions[i].
template <class Ser>
inline void put_batch_proof(Ser& s, const std::vector<size_t>& positions, const std::vector<const u32*>& raw, u32 h) {
    s.u64le(positions.size());
    for (size_t p : positions) s.u32le((u32)p);
    s.u64le(positions.size());
    for (const u32* r : raw) s.u32le(r[0]);
    // (node index at the current level, a position that lies below it), ascending and unique
    std::vector<std::pair<size_t, size_t>> known, next;
    known.reserve(positions.size());
    for (size_t i = 0; i < positions.size(); i++) known.emplace_back(positions[i], i);
    std::sort(known.begin(), known.end());
    known.erase(std::unique(known.begin(), known.end(), [](auto& a, auto& b) { return a.first == b.first; }), known.end());
    s.u64le(h);
    std::vector<const u32*> lvl;
    for (u32 k = 0; k < h; k++) {
        lvl.clear();
        next.clear();
        for (size_t i = 0; i < known.size(); i++) {
            const size_t node = known[i].first;
            // the sibling, if known, is the neighbour in the sorted list
            const bool sib_known = (node & 1) ? (i > 0 && known[i - 1].first == node - 1) : (i + 1 < known.size() && known[i + 1].first == node + 1);
            if (!sib_known) lvl.push_back(k == 0 ? raw[known[i].second] + 1 : raw[known[i].second] + 2 + 4 * (size_t)(k - 1));
            if (next.empty() || next.back().first != (node >> 1)) next.emplace_back(node >> 1, known[i].second);
        }
        s.u64le(lvl.size());
        for (const u32* d : lvl) {
            if (k == 0) { s.u32le(d[0]); s.u32le(0); s.u32le(0); s.u32le(0); }     // hash_leaf of the sibling value
            else { s.u32le(d[0]); s.u32le(d[1]); s.u32le(d[2]); s.u32le(d[3]); }
        }
        known.swap(next);
    }
}
template <class Ser>
inline void put_digest(Ser& s, const u32* d) { for (int i = 0; i < 4; i++) s.u32le(d[i]); }

// bincode(BasefoldCommitment) (basefold.rs:39-47)
template <class Ser>
inline void put_basefold_commitment(Ser& s, const u32* rec_host, const BfPending& pd) {
    put_digest(s, rec_host + pd.root_off);
    s.u64le(pd.num_coeffs);
    s.u64le(pd.log_n);
}
// bincode(BasefoldOpeningProof) (basefold.rs:50-64)
template <class Ser>
inline void put_basefold_proof(Ser& s, const u32* rec_host, const BfPending& pd) {
    const u32 log_n = pd.log_n;
    s.u64le(log_n);
    for (u32 r = 0; r < log_n; r++) put_digest(s, rec_host + pd.round_off[r]);
    s.u64le(log_n);
    for (u32 r = 0; r < log_n; r++) {
        const u32 h_prev = log_n + 1 - r, h_fold = h_prev - 1;
        const u32* rec = rec_host + pd.round_off[r];
        const u32* idx = rec + 4;
        const size_t prev_half = size_t(1) << (h_prev - 1);
        const size_t pw_prev = 2 + 4 * (size_t)(h_prev - 1), pw_fold = 2 + 4 * (size_t)(h_fold - 1);
        const u32* out_prev = rec + 4 + BF_QUERIES;
        const u32* out_fold = out_prev + 2 * BF_QUERIES * pw_prev;
        std::vector<size_t> pp, fp;
        std::vector<const u32*> pr, fr;
        for (u32 q = 0; q < BF_QUERIES; q++) {
            pp.push_back(idx[q]); pr.push_back(out_prev + (2 * q) * pw_prev);
            pp.push_back(idx[q] + prev_half); pr.push_back(out_prev + (2 * q + 1) * pw_prev);
            fp.push_back(idx[q]); fr.push_back(out_fold + q * pw_fold);
        }
        put_batch_proof(s, pp, pr, h_prev);
        put_batch_proof(s, fp, fr, h_fold);
    }
    s.u32le(rec_host[pd.final_off]);
    s.u64le(0);                                   // final_coeffs: empty
}

}  // namespace zkb
