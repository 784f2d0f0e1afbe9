// Merkle trees with 16-byte digests over vectors of field elements
// (rust/zk_ml_prover/src/proving/pcs.rs:57-196).
//
//   leaf      u32 value, little-endian, zero-padded to 16 bytes, not hashed      pcs.rs:71-75
//   node      blake3(L || R) truncated to 16 bytes (what the reference computes   pcs.rs:125-134
//             on every target except aarch64), or the AES-based Matyas-Meyer-
//             Oseas compression it uses on aarch64                               pcs.rs:92-121
//
// A tree of height h over 2^h leaves stores layers 1..h (layer k has 2^(h-k) nodes) back to
// back: layer k starts at node offset 2^h - 2^(h-k+1); the root is node 2^h - 2.  One launch
// of mk_tile_kernel builds up to MK_TILE_LOG levels: each CTA owns MK_TILE consecutive inputs,
// keeps the running level in shared memory and writes every level it produces; levels of 2^20 inputs
// and more go to mk_lane_kernel, four at a time.  A 32-byte node
// input is a single blake3 block, so one node costs one compression; the kernel is bound by
// integer issue, not by bandwidth (16 bytes read and 8 written per compression on average).
#pragma once
#include "blake3.cuh"

namespace zkb {

enum NodeHash : int { NODE_BLAKE3 = 0, NODE_AES_MMO = 1 };

// ---- blake3 node: one block of 32 bytes, flags CHUNK_START | CHUNK_END | ROOT -------------------
// Message words 8..15 are zero, so with the schedule resolved at compile time half of the
// message additions disappear; over two leaves (LEAVES) only words 0 and 4 are not zero.
template <bool LEAVES = false>
__device__ __forceinline__ uint4 b3_node(uint4 l, uint4 r) {
    u32 w[16] = {l.x, l.y, l.z, l.w, r.x, r.y, r.z, r.w, 0, 0, 0, 0, 0, 0, 0, 0};
    if (LEAVES) w[1] = w[2] = w[3] = w[5] = w[6] = w[7] = 0;
    u32 s0 = 0x6a09e667u, s1 = 0xbb67ae85u, s2 = 0x3c6ef372u, s3 = 0xa54ff53au;
    u32 s4 = 0x510e527fu, s5 = 0x9b05688cu, s6 = 0x1f83d9abu, s7 = 0x5be0cd19u;
    u32 s8 = 0x6a09e667u, s9 = 0xbb67ae85u, s10 = 0x3c6ef372u, s11 = 0xa54ff53au;
    u32 s12 = 0, s13 = 0, s14 = 32, s15 = B3_CHUNK_START | B3_CHUNK_END | B3_ROOT;
#pragma unroll
    for (int rd = 0; rd < 7; rd++) {
        B3_G(s0, s4, s8, s12, w[0], w[1]);   B3_G(s1, s5, s9, s13, w[2], w[3]);
        B3_G(s2, s6, s10, s14, w[4], w[5]);  B3_G(s3, s7, s11, s15, w[6], w[7]);
        B3_G(s0, s5, s10, s15, w[8], w[9]);  B3_G(s1, s6, s11, s12, w[10], w[11]);
        B3_G(s2, s7, s8, s13, w[12], w[13]); B3_G(s3, s4, s9, s14, w[14], w[15]);
        if (rd < 6) {
            u32 t[16] = {w[2], w[6], w[3], w[10], w[7], w[0], w[4], w[13], w[1], w[11], w[12], w[5], w[9], w[14], w[15], w[8]};
#pragma unroll
            for (int i = 0; i < 16; i++) w[i] = t[i];
        }
    }
    return make_uint4(s0 ^ s8, s1 ^ s9, s2 ^ s10, s3 ^ s11);
}

// ---- AES-MMO node -------------------------------------------------------------------------------
// ARM's AESE is AddRoundKey, SubBytes, ShiftRows (in that order) and AESMC is MixColumns; the
// reference runs ten AESE steps keyed L, R, L, R, ... on the state L^R, MixColumns after the
// first nine, and XORs L^R back in.  SubBytes + ShiftRows + MixColumns of one column is four
// lookups in a table T0[x] = (2 S[x], S[x], S[x], 3 S[x]) and byte rotations of it.
__constant__ u32 AES_T0[256];
__constant__ unsigned char AES_SBOX[256];

struct AesTables { u32 t0[256]; unsigned char sbox[256]; };
// S-box from its definition (FIPS-197 5.1.1): inverse in GF(2^8) mod x^8+x^4+x^3+x+1, then the affine map.
inline AesTables aes_make_tables() {
    AesTables t;
    auto xt = [](unsigned a) { return ((a << 1) ^ ((a & 0x80) ? 0x11b : 0)) & 0xff; };
    auto mul = [&](unsigned a, unsigned b) { unsigned r = 0; while (b) { if (b & 1) r ^= a; a = xt(a); b >>= 1; } return r; };
    for (unsigned x = 0; x < 256; x++) {
        unsigned inv = 0;
        if (x) { inv = 1; for (int i = 0; i < 254; i++) inv = mul(inv, x); }
        unsigned s = inv;
        for (int i = 1; i <= 4; i++) s ^= ((inv << i) | (inv >> (8 - i))) & 0xff;
        s ^= 0x63;
        t.sbox[x] = (unsigned char)s;
        unsigned s2 = xt(s), s3 = s2 ^ s;
        t.t0[x] = s2 | (s << 8) | (s << 16) | (s3 << 24);
    }
    return t;
}

__device__ __forceinline__ u32 rotl8(u32 x, int bytes) { return __funnelshift_l(x, x, 8 * bytes); }
__device__ __forceinline__ uint4 aes_node(uint4 l, uint4 r, const u32* __restrict__ T0, const unsigned char* __restrict__ S) {
    const u32 x0 = l.x ^ r.x, x1 = l.y ^ r.y, x2 = l.z ^ r.z, x3 = l.w ^ r.w;
    u32 c0 = x0, c1 = x1, c2 = x2, c3 = x3;
#pragma unroll
    for (int rd = 0; rd < 10; rd++) {
        const uint4 k = (rd & 1) ? r : l;
        c0 ^= k.x; c1 ^= k.y; c2 ^= k.z; c3 ^= k.w;
        u32 n0, n1, n2, n3;
        if (rd < 9) {
            n0 = T0[c0 & 255] ^ rotl8(T0[(c1 >> 8) & 255], 1) ^ rotl8(T0[(c2 >> 16) & 255], 2) ^ rotl8(T0[c3 >> 24], 3);
            n1 = T0[c1 & 255] ^ rotl8(T0[(c2 >> 8) & 255], 1) ^ rotl8(T0[(c3 >> 16) & 255], 2) ^ rotl8(T0[c0 >> 24], 3);
            n2 = T0[c2 & 255] ^ rotl8(T0[(c3 >> 8) & 255], 1) ^ rotl8(T0[(c0 >> 16) & 255], 2) ^ rotl8(T0[c1 >> 24], 3);
            n3 = T0[c3 & 255] ^ rotl8(T0[(c0 >> 8) & 255], 1) ^ rotl8(T0[(c1 >> 16) & 255], 2) ^ rotl8(T0[c2 >> 24], 3);
        } else {
            n0 = (u32)S[c0 & 255] | ((u32)S[(c1 >> 8) & 255] << 8) | ((u32)S[(c2 >> 16) & 255] << 16) | ((u32)S[c3 >> 24] << 24);
            n1 = (u32)S[c1 & 255] | ((u32)S[(c2 >> 8) & 255] << 8) | ((u32)S[(c3 >> 16) & 255] << 16) | ((u32)S[c0 >> 24] << 24);
            n2 = (u32)S[c2 & 255] | ((u32)S[(c3 >> 8) & 255] << 8) | ((u32)S[(c0 >> 16) & 255] << 16) | ((u32)S[c1 >> 24] << 24);
            n3 = (u32)S[c3 & 255] | ((u32)S[(c0 >> 8) & 255] << 8) | ((u32)S[(c1 >> 16) & 255] << 16) | ((u32)S[c2 >> 24] << 24);
        }
        c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    }
    return make_uint4(c0 ^ x0, c1 ^ x1, c2 ^ x2, c3 ^ x3);
}

// The same node with T0 replicated once per bank, so that the lookups of a warp never meet in one: word x * 32 + b
// of `rep` is T0[x], lane b reads column b.  With one copy a lookup takes the warp three to four passes.  The
// last round's S[x] is the second byte of T0[x].
constexpr int AES_REP_WORDS = 256 * 32;
__device__ __forceinline__ void aes_rep_fill(u32* rep) {
    for (u32 i = threadIdx.x; i < (u32)AES_REP_WORDS; i += blockDim.x) rep[i] = AES_T0[i >> 5];
}
template <int BYTE>
__device__ __forceinline__ u32 aes_rep_at(const u32* __restrict__ rep, u32 lane4, u32 c) {
    const u32 sh = BYTE == 0 ? c << 7 : c >> (8 * BYTE - 7);
    return *reinterpret_cast<const u32*>(reinterpret_cast<const unsigned char*>(rep) + ((sh & 0x7f80u) | lane4));
}
__device__ __forceinline__ u32 aes_rep_column(const u32* __restrict__ rep, u32 l4, u32 a, u32 b, u32 c, u32 d) {
    return aes_rep_at<0>(rep, l4, a) ^ rotl8(aes_rep_at<1>(rep, l4, b), 1) ^ rotl8(aes_rep_at<2>(rep, l4, c), 2) ^ rotl8(aes_rep_at<3>(rep, l4, d), 3);
}
__device__ __forceinline__ u32 aes_rep_last(const u32* __restrict__ rep, u32 l4, u32 a, u32 b, u32 c, u32 d) {
    const u32 lo = __byte_perm(aes_rep_at<0>(rep, l4, a), aes_rep_at<1>(rep, l4, b), 0x0051);
    const u32 hi = __byte_perm(aes_rep_at<2>(rep, l4, c), aes_rep_at<3>(rep, l4, d), 0x0051);
    return __byte_perm(lo, hi, 0x5410);
}
__device__ __forceinline__ uint4 aes_node_rep(uint4 l, uint4 r, const u32* __restrict__ rep) {
    const u32 l4 = (threadIdx.x & 31) * 4;
    const u32 x0 = l.x ^ r.x, x1 = l.y ^ r.y, x2 = l.z ^ r.z, x3 = l.w ^ r.w;
    u32 c0 = x0, c1 = x1, c2 = x2, c3 = x3;
#pragma unroll
    for (int rd = 0; rd < 10; rd++) {
        const uint4 k = (rd & 1) ? r : l;
        c0 ^= k.x; c1 ^= k.y; c2 ^= k.z; c3 ^= k.w;
        u32 n0, n1, n2, n3;
        if (rd < 9) {
            n0 = aes_rep_column(rep, l4, c0, c1, c2, c3); n1 = aes_rep_column(rep, l4, c1, c2, c3, c0);
            n2 = aes_rep_column(rep, l4, c2, c3, c0, c1); n3 = aes_rep_column(rep, l4, c3, c0, c1, c2);
        } else {
            n0 = aes_rep_last(rep, l4, c0, c1, c2, c3); n1 = aes_rep_last(rep, l4, c1, c2, c3, c0);
            n2 = aes_rep_last(rep, l4, c2, c3, c0, c1); n3 = aes_rep_last(rep, l4, c3, c0, c1, c2);
        }
        c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    }
    return make_uint4(c0 ^ x0, c1 ^ x1, c2 ^ x2, c3 ^ x3);
}

// ---- tree storage ---------------------------------------------------------------------------------
__host__ __device__ __forceinline__ size_t mk_layer_offset(u32 h, u32 k) { return (size_t(1) << h) - (size_t(1) << (h - k + 1)); }
__host__ __device__ __forceinline__ size_t mk_node_count(u32 h) { return (size_t(1) << h) - 1; }

constexpr int MK_TILE_LOG = 10;
constexpr int MK_TILE = 1 << MK_TILE_LOG;
constexpr int MK_THREADS = 256;

// How a CTA obtains its MK_TILE inputs.
enum MkMode : int {
    MK_VALUES = 0,   // u32 leaves (zero beyond n_valid)
    MK_DIGESTS = 1,  // nodes of layer k0 of the same tree
    MK_FOLD = 2      // leaves produced on the fly by a Basefold codeword fold (see basefold.cuh)
};

struct MkFold {
    const u32* prev;      // previous codeword, 2 * half values
    u32* out;             // folded codeword, half values
    const u32* weights;   // w_level of this fold, w_len values
    const u32* alpha;     // device-resident challenge
    u32* eval_src;        // coefficient buffer being evaluated (eval_half * 2 live values), or null
    u32* eval_dst;        // where the folded coefficients go (may equal eval_src)
    size_t w_len, eval_half;
    // batch openings: values added to the folded codeword before it is stored and hashed (the already scaled sum of the
    // codewords that join the chain at this length), or null
    const u32* add; size_t add_mask;      // add[j & add_mask]: a joining codeword is [v || v], only v is summed
    // prev[j + prev_partner] is the other value of a pair: half of the codeword's length, or 0 while the codeword is
    // [c || c] and only c is stored (its two values are then the same, and the fold leaves c as it is)
    size_t prev_partner;
    int doubled;          // the launch that reaches the root also stores the node over (root, root) behind it: the root of [c || c]
};

__device__ __forceinline__ u32 coef_at(const u32* __restrict__ p, u32 rows, u32 cols, u32 log_cols_pad, size_t i) {
    size_t r = i >> log_cols_pad, c = i & ((size_t(1) << log_cols_pad) - 1);
    return (r < rows && c < cols) ? p[r * cols + c] : 0u;
}

// One value of the folded codeword (and, below eval_half, of the folded coefficients).
__device__ __forceinline__ u32 mk_fold_value(const MkFold& fold, Fp alpha, size_t j) {
    const Fp two_inv{1073741824u};
    Fp l{fold.prev[j]}, r{fold.prev[j + fold.prev_partner]};
    Fp w{fold.weights[j & (fold.w_len - 1)]};
    Fp f = (l + r) * two_inv + alpha * ((l - r) * w);
    if (fold.add) f = f + Fp{fold.add[j & fold.add_mask]};
    fold.out[j] = f.v;
    if (fold.eval_dst && j < fold.eval_half) {
        const Fp a{fold.eval_src[j]}, b{fold.eval_src[j + fold.eval_half]};
        fold.eval_dst[j] = ((fp_one() - alpha) * a + alpha * b).v;
    }
    return f.v;
}

// One CTA: MK_TILE inputs (fewer when the whole level is smaller) -> up to MK_TILE_LOG layers.
// n_in = number of inputs at level k0 (a power of two); h = height of the tree.  DOUBLED (the launch that reaches the root of a
// half codeword's tree) stores the node over (root, root) behind the root.  It is a variant of its own because as a condition at run
// time it costs the other launches: the AES leaf variant gets 32 registers instead of 36, and on B200 a call for the root of 1024
// values took 44.1 us instead of 36.5.
template <int KIND, int MODE, bool DOUBLED>
__global__ void __launch_bounds__(MK_THREADS) mk_tile_kernel(const u32* __restrict__ values, size_t n_valid, size_t n_in, u32 k0, u32 h,
                                                            uint4* __restrict__ nodes, MkFold fold) {
    __shared__ uint4 bufA[MK_TILE];
    __shared__ uint4 bufB[MK_TILE / 2];
    __shared__ u32 t0_s[KIND == NODE_AES_MMO ? 256 : 1];
    __shared__ unsigned char sb_s[KIND == NODE_AES_MMO ? 256 : 1];
    if (KIND == NODE_AES_MMO) {
        for (int i = threadIdx.x; i < 256; i += MK_THREADS) { t0_s[i] = AES_T0[i]; sb_s[i] = AES_SBOX[i]; }
    }
    const size_t tile = n_in < (size_t)MK_TILE ? n_in : (size_t)MK_TILE;
    const size_t base = (size_t)blockIdx.x * tile;

    if (MODE == MK_DIGESTS) {
        const uint4* in = nodes + mk_layer_offset(h, k0) + base;
        for (size_t i = threadIdx.x; i < tile; i += MK_THREADS) bufA[i] = in[i];
    } else if (MODE == MK_VALUES) {
        for (size_t i = threadIdx.x; i < tile; i += MK_THREADS) {
            size_t g = base + i;
            bufA[i] = make_uint4(g < n_valid ? values[g] : 0u, 0, 0, 0);
        }
    } else {
        const Fp alpha{*fold.alpha};
        for (size_t i = threadIdx.x; i < tile; i += MK_THREADS) bufA[i] = make_uint4(mk_fold_value(fold, alpha, base + i), 0, 0, 0);
    }
    __syncthreads();

    uint4* cur = bufA;
    uint4* nxt = bufB;
    size_t cnt = tile;
    u32 k = k0;
    while (cnt > 1 && k < h) {
        const size_t out_cnt = cnt >> 1;
        k++;
        uint4* layer = nodes + mk_layer_offset(h, k) + (size_t)blockIdx.x * out_cnt;
        for (size_t i = threadIdx.x; i < out_cnt; i += MK_THREADS) {
            uint4 d = KIND == NODE_AES_MMO ? aes_node(cur[2 * i], cur[2 * i + 1], t0_s, sb_s) : b3_node(cur[2 * i], cur[2 * i + 1]);
            nxt[i] = d;
            layer[i] = d;
        }
        __syncthreads();
        uint4* t = cur; cur = nxt; nxt = t;
        cnt = out_cnt;
    }
    if (DOUBLED && threadIdx.x == 0)
        nodes[mk_node_count(h)] = KIND == NODE_AES_MMO ? aes_node(cur[0], cur[0], t0_s, sb_s) : b3_node(cur[0], cur[0]);
}

// Four levels of a level that is large enough to give every thread a subtree of its own: 16 consecutive inputs, their
// fifteen nodes one after the other in post-order, the nodes that wait for their sibling in registers.  No lane is ever
// idle and no barrier separates the levels; in a tile the last five levels run on part of a warp, and most warps wait.
// Leaves are staged (and folded) through shared memory with coalesced accesses, one word of padding per thread.
// Bound by integer issue (ncu: ALU pipe 90 % busy, DRAM 3 %): 34.6 G blake3 nodes/s over 2^24 leaves, 33.2 G AES nodes/s, where the
// tile kernel reached 26.9 G blake3 nodes/s and the node alone runs at 37.  Measured on B200 with the tile kernel -> with this
// one at the top: Basefold of 2^24 coefficients 3475 -> 3213 us (blake3), a batch of seven polynomials up to 2^22 2682 -> 2452 us
// (AES).  Below 2^20 inputs there are fewer than 2^16 subtrees, not four warps to a scheduler, and fifteen nodes in a row would
// take longer than a tile's ten levels.
constexpr int MK_LANE_LOG = 4, MK_LANE = 1 << MK_LANE_LOG, MK_LANE_THREADS = 256;
constexpr size_t mk_lane_smem(int kind) { return kind == NODE_AES_MMO ? AES_REP_WORDS * 4 : 0; }
constexpr size_t MK_LANE_MIN = size_t(1) << 20;      // inputs: below, the subtrees are too few to fill the GPU
template <int KIND, int MODE>
__global__ void __launch_bounds__(MK_LANE_THREADS) mk_lane_kernel(const u32* __restrict__ values, size_t n_valid, u32 k0, u32 h,
                                                                 uint4* __restrict__ nodes, MkFold fold) {
    __shared__ u32 leaf[MODE == MK_DIGESTS ? 1 : MK_LANE_THREADS * (MK_LANE + 1)];
    extern __shared__ __align__(16) u32 rep[];               // AES: the replicated table (mk_lane_smem bytes)
    if (KIND == NODE_AES_MMO) aes_rep_fill(rep);
    const size_t base = (size_t)blockIdx.x * (MK_LANE_THREADS * MK_LANE);
    if (MODE != MK_DIGESTS) {
        Fp alpha{0};
        if (MODE == MK_FOLD) alpha.v = *fold.alpha;
        for (u32 e = threadIdx.x; e < MK_LANE_THREADS * MK_LANE; e += MK_LANE_THREADS) {
            const size_t g = base + e;
            u32 v;
            if (MODE == MK_FOLD) v = mk_fold_value(fold, alpha, g);
            else v = g < n_valid ? values[g] : 0u;
            leaf[e + (e >> MK_LANE_LOG)] = v;
        }
    }
    __syncthreads();
    const size_t t = base / MK_LANE + threadIdx.x;          // this thread's node four levels up
    const u32* mine = leaf + threadIdx.x * (MK_LANE + 1);
    const uint4* in = MODE == MK_DIGESTS ? nodes + mk_layer_offset(h, k0) + t * MK_LANE : nullptr;
    uint4 w1 = make_uint4(0, 0, 0, 0), w2 = w1, w3 = w1, d = w1;       // waiting nodes of levels 1..3
    u32 pair = 0, lvl = 0;
    while (lvl < MK_LANE_LOG) {                              // the same for all threads
        if (MODE != MK_DIGESTS && lvl == 0) {
            const uint4 l = make_uint4(mine[2 * pair], 0, 0, 0), r = make_uint4(mine[2 * pair + 1], 0, 0, 0);
            d = KIND == NODE_AES_MMO ? aes_node_rep(l, r, rep) : b3_node<true>(l, r);
        } else {
            uint4 l, r = d;
            if (lvl == 0) { l = in[2 * pair]; r = in[2 * pair + 1]; }
            else l = lvl == 1 ? w1 : (lvl == 2 ? w2 : w3);
            d = KIND == NODE_AES_MMO ? aes_node_rep(l, r, rep) : b3_node(l, r);
        }
        const u32 q = pair >> lvl;                           // index of the node within this thread's nodes of its level
        lvl++;
        nodes[mk_layer_offset(h, k0 + lvl) + (t << (MK_LANE_LOG - lvl)) + q] = d;
        if (lvl < MK_LANE_LOG && !(q & 1)) {                 // a left child waits; the next pair of inputs follows
            if (lvl == 1) w1 = d; else if (lvl == 2) w2 = d; else w3 = d;
            lvl = 0;
            pair++;
        }
    }
}

// Raw authentication data of opened positions: for position p of a tree of height h over
// `values`, out = [value, sibling value, sibling digest at level 1, ..., level h-1] (2 + 4 (h-1)
// words).  The host drops the digests a batch proof does not need (pcs.rs:290-337).
__device__ inline void mk_gather_path(const u32* __restrict__ values, size_t n_valid, const uint4* __restrict__ nodes, u32 h, size_t p,
                                      u32* out, int lane, int nlanes) {
    for (u32 k = lane; k <= h; k += nlanes) {
        if (k == 0) {
            out[0] = p < n_valid ? values[p] : 0u;
        } else if (k == 1) {
            size_t s = p ^ 1;
            out[1] = s < n_valid ? values[s] : 0u;
        } else {
            size_t s = (p >> (k - 1)) ^ 1;
            uint4 d = nodes[mk_layer_offset(h, k - 1) + s];
            u32* o = out + 2 + 4 * (size_t)(k - 2);
            o[0] = d.x; o[1] = d.y; o[2] = d.z; o[3] = d.w;
        }
    }
}
// The same path out of the tree of height h + 1 over [v || v], of which the tree of height h over v is stored: below the
// root both halves have the same nodes, and the last sibling is the other half's root, which is the stored one.
__device__ inline void mk_gather_path_doubled(const u32* __restrict__ values, const uint4* __restrict__ nodes, u32 h, size_t p, u32* out,
                                              int lane, int nlanes) {
    const size_t n = size_t(1) << h;
    mk_gather_path(values, n, nodes, h, p & (n - 1), out, lane, nlanes);
    if (lane == 0) {
        const uint4 d = nodes[mk_layer_offset(h, h)];
        u32* o = out + 2 + 4 * (size_t)(h - 1);
        o[0] = d.x; o[1] = d.y; o[2] = d.z; o[3] = d.w;
    }
}
// Positions given by the host (the stand-alone Merkle entry points).
__global__ void mk_open_kernel(const u32* __restrict__ values, size_t n_valid, const uint4* __restrict__ nodes, u32 h,
                               const unsigned long long* __restrict__ pos, u32 n_pos, u32* out) {
    for (u32 q = blockIdx.x; q < n_pos; q += gridDim.x)
        mk_gather_path(values, n_valid, nodes, h, (size_t)pos[q], out + (size_t)q * (2 + 4 * (size_t)(h - 1)), threadIdx.x, blockDim.x);
}

}  // namespace zkb
