// Single-CTA tail of the product sumcheck, over EF tables with EF challenges or over base-field tables with base-field
// challenges (T = Fe or Fp), with the table work taken off the critical path
// (rust/zk_ml_prover/src/proving/sumcheck.rs:211-272, 1262-1315 compute the same messages).
//
// In the plain tail every round is: pass over the tables (fold with the last challenge, sum the
// round polynomial), block reduction, then one warp hashes (about five SHA-256 compressions, a second warp beside it)
// while thirty wait.  Here warp 0 only hashes.  While it hashes round k, the other warps
// fold the tables with r_(k-1) and compute the NEXT round's sums as polynomials in the still
// unknown r_k: with lo(r) = a + r (b - a), hi(r) = c + r (d - c) over the four quarters a, b, c,
// d of a table, each of s0 = sum lo_f lo_g, s1 = sum hi_f hi_g, s2 = sum (2hi - lo)_f (2hi - lo)_g
// is a quadratic in r with nine EF coefficient sums in all.  When r_k arrives the hashing thread
// evaluates the three quadratics and goes on hashing; the table work overlaps the hash chain
// instead of alternating with it.  All values are canonical field elements, so the messages are
// bit-identical to the plain tail's.
// Base-field rounds hash one compression instead of five, so the table pass and its reduction were most of such a round:
// measured on B200 with the plain tail -> with this one, a whole op-list proof of the 1024-2048-1024-10 MLP 1676 -> 1579 us,
// of the 182-op GPT-2 shape 60.6 -> 57.3 ms.
#pragma once
#include "sumcheck.cuh"

namespace zkb {

constexpr int PIPE_THREADS = 512;                                 // at most; 128 registers per thread (the worker pass keeps 36 sums)
constexpr int PIPE_MAX_WORKER_WARPS = PIPE_THREADS / 32 - 1;      // 15
template <class T> constexpr int PIPE_NW = 9 * Width<T>::W;   // nine coefficient sums

// Roles.  Warp 0 hashes.  Warps 4, 8, 12 would share warp 0's scheduler (warp w issues on sub-
// partition w mod 4), its instruction cache and its issue slots; they only join the CTA barriers,
// so the hash chain has a sub-partition to itself.  While a round's tables are long its table pass takes longer than its
// hash, and all other warps are workers.  From pipe_paired() on warp 1 expands the message schedules instead (TrPair), with the
// second sub-partition to itself, and the warps of the other two are the workers.  They are numbered 0, 1, 2, ... in warp order.
struct PipeRole { int index, warps; };           // index below 0: not a worker
__device__ __forceinline__ PipeRole pipe_role(bool paired) {
    const int warp = threadIdx.x >> 5, n = blockDim.x >> 5;
    if (!paired) return PipeRole{(warp & 3) ? warp - 1 - (warp >> 2) : -1, n - 1 - ((n - 1) >> 2)};
    return PipeRole{(warp & 3) >= 2 ? 2 * (warp >> 2) + (warp & 3) - 2 : -1, 2 * (n >> 2) + ((n & 3) == 3 ? 1 : 0)};
}
// n: length of the tables whose message a round hashes.  The line lies where the pass of the workers that are left takes about as
// long as the shared hash.  Measured on B200, never paired / this line / always: four 4B-shape layers 16.77 / 16.20 / 16.31 ms, the
// 1024-2048-1024-10 MLP (base field) 1384 / 1352 / 1352 us.
template <class T> __device__ __forceinline__ bool pipe_paired(size_t n) {
    return n <= (Width<T>::W == 4 ? 128 : 512) * (size_t)(blockDim.x >> 5);
}
// Barrier 1 among the worker warps only.
__device__ __forceinline__ void pipe_worker_barrier(int warps) { asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory"); }

// Coefficient sums of the next round over one pair index: quarters (a, b, c, d) of f and g.
template <class T>
__device__ __forceinline__ void pipe_accum(T* C, T fa, T fb, T fc, T fd, T ga, T gb, T gc, T gd) {
    const T ef = fb - fa, eg = gb - ga, hf = fd - fc, hg = gd - gc;       // lo = a + r e, hi = c + r h
    C[0] = C[0] + fa * ga;  C[1] = C[1] + fa * eg + ga * ef;  C[2] = C[2] + ef * eg;
    C[3] = C[3] + fc * gc;  C[4] = C[4] + fc * hg + gc * hf;  C[5] = C[5] + hf * hg;
    const T pf = dbl_minus(fc, fa), pg = dbl_minus(gc, ga);               // 2 hi - lo at r = 0
    const T qf = dbl_minus(hf, ef), qg = dbl_minus(hg, eg);               // its slope in r
    C[6] = C[6] + pf * pg;  C[7] = C[7] + pf * qg + pg * qf;  C[8] = C[8] + qf * qg;
}

// Workers only.  Tables of size n at (rf, rg); if `fold`, they are first
// folded with r into size n / 2 at (wf, wg) (in place allowed) and the sums are taken over the
// folded tables.  Leaves the PIPE_NW summed words in out[] (shared memory) when the result size is >= 4.
template <class T>
__device__ __forceinline__ void pipe_worker_pass(const T* rf, const T* rg, T* wf, T* wg, size_t n, bool fold, T r,
                                                 u32 (*cw)[PIPE_NW<T>], u32* out, PipeRole role) {
    constexpr int NW = PIPE_NW<T>;
    const int worker_warps = role.warps;
    const int wid = role.index * 32 + (threadIdx.x & 31);
    const size_t workers = (size_t)worker_warps * 32;
    const size_t m = fold ? n / 2 : n;              // size of the tables the sums run over
    T C[9];
#pragma unroll
    for (int i = 0; i < 9; i++) C[i] = zero_of<T>();
    if (m >= 4) {
        const size_t q = m / 4;                     // pair indices of the next round
        for (size_t j = wid; j < q; j += workers) {
            T fa, fb, fc, fd, ga, gb, gc, gd;
            if (fold) {
                // folded element x is lerp(T[x], T[x + n/2], r); this thread owns x = j, j+q, j+2q, j+3q
                const size_t h = n / 2;
                fa = lerp(ld_fe(rf + j), ld_fe(rf + j + h), r);                 ga = lerp(ld_fe(rg + j), ld_fe(rg + j + h), r);
                fc = lerp(ld_fe(rf + j + q), ld_fe(rf + j + q + h), r);         gc = lerp(ld_fe(rg + j + q), ld_fe(rg + j + q + h), r);
                fb = lerp(ld_fe(rf + j + 2 * q), ld_fe(rf + j + 2 * q + h), r); gb = lerp(ld_fe(rg + j + 2 * q), ld_fe(rg + j + 2 * q + h), r);
                fd = lerp(ld_fe(rf + j + 3 * q), ld_fe(rf + j + 3 * q + h), r); gd = lerp(ld_fe(rg + j + 3 * q), ld_fe(rg + j + 3 * q + h), r);
                st_fe(wf + j, fa); st_fe(wf + j + q, fc); st_fe(wf + j + 2 * q, fb); st_fe(wf + j + 3 * q, fd);
                st_fe(wg + j, ga); st_fe(wg + j + q, gc); st_fe(wg + j + 2 * q, gb); st_fe(wg + j + 3 * q, gd);
            } else {
                fa = ld_fe(rf + j); fc = ld_fe(rf + j + q); fb = ld_fe(rf + j + 2 * q); fd = ld_fe(rf + j + 3 * q);
                ga = ld_fe(rg + j); gc = ld_fe(rg + j + q); gb = ld_fe(rg + j + 2 * q); gd = ld_fe(rg + j + 3 * q);
            }
            pipe_accum(C, fa, fb, fc, fd, ga, gb, gc, gd);
        }
    } else if (fold) {
        // two elements remain after this fold: nothing to sum, just fold (one thread)
        if (wid == 0) {
            const size_t h = n / 2;
            for (size_t x = 0; x < h; x++) {
                T a = lerp(ld_fe(rf + x), ld_fe(rf + x + h), r), b = lerp(ld_fe(rg + x), ld_fe(rg + x + h), r);
                st_fe(wf + x, a); st_fe(wg + x, b);
            }
        }
    }
    if (m >= 4) {
        u32 w[NW];
#pragma unroll
        for (int i = 0; i < 9; i++) to_words(C[i], w + Width<T>::W * i);
        const int lane = threadIdx.x & 31, warp = role.index;
#pragma unroll
        for (int k = 0; k < NW; k++) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) w[k] = add31(w[k], __shfl_down_sync(0xffffffffu, w[k], off));
        }
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < NW; k++) cw[warp][k] = w[k];
        }
        pipe_worker_barrier(worker_warps);
        for (int k = wid; k < NW; k += (int)workers) {
            u32 v = 0;
            for (int rw = 0; rw < worker_warps; rw++) v = add31(v, cw[rw][k]);
            out[k] = v;
        }
    }
}

template <class T>
__global__ void __launch_bounds__(PIPE_THREADS) sc_tail_product_pipe_kernel(ScTables tb, size_t size, u32 round, u32 num_vars,
                                                                               int pending, ScIO io) {
    pdl_small_prologue();
    constexpr int W = Width<T>::W, NW = PIPE_NW<T>;
    __shared__ u32 red[32 * 16];
    __shared__ __align__(16) unsigned char trbuf[TR_SCRATCH_BYTES];
    __shared__ u32 r_sh[2][W];                       // indexed by round parity: round k+1's challenge never overwrites r_k while a slow warp still reads it
    __shared__ u32 cw[PIPE_MAX_WORKER_WARPS][NW];
    __shared__ u32 csum[2][NW];
    __shared__ u32 w_sh[3 * W];

    ZKB_STAMP_BEGIN
    const int warp = threadIdx.x >> 5;
    TrPair tr;
    if (warp == 0) tr_load(tr, io.tr, trbuf);
    T r = zero_of<T>();
    if (pending) from_words(r, io.chal + (size_t)(round - 1) * W);

    // ---- prologue: the message of `round`, computed directly by the whole CTA
    const T* rf = reinterpret_cast<const T*>(tb.src[0]);
    const T* rg = reinterpret_cast<const T*>(tb.src[1]);
    T* wf = reinterpret_cast<T*>(tb.dst[0]);
    T* wg = reinterpret_cast<T*>(tb.dst[1]);
    size_t n = size;                                 // size of the tables the current round sums over
    u32 w[16];
    {
        T acc[3] = {zero_of<T>(), zero_of<T>(), zero_of<T>()};
        if (pending) {
            sc_pass<SC_PRODUCT, T, T, true>(tb, n / 4, r, threadIdx.x, blockDim.x, acc);
            n /= 2;
            rf = wf; rg = wg;                        // folded tables live in dst from now on
        } else {
            sc_pass<SC_PRODUCT, T, T, false>(tb, n / 2, r, threadIdx.x, blockDim.x, acc);
        }
#pragma unroll
        for (int k = 0; k < 3; k++) to_words(acc[k], w + W * k);
        block_sum_words<3 * W>(w, red);                 // ends with a CTA barrier: folded tables visible
    }

    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < 3 * W; i++) w[i] = __shfl_sync(0xffffffffu, w[i], 0);
    }
    bool first = true;
    u32 k = round;
    for (;;) {
        // warp 0 hashes round k; the workers prepare round k + 1 as polynomials in r_k
        const bool paired = pipe_paired<T>(n);
        const PipeRole role = pipe_role(paired);
        if (warp == 0) {
            T rn;
            if (paired) {
                rn = sc_finish_round<SC_PRODUCT, T, T>(w, io, k, tr);
                tr_pair_end(tr);
            } else rn = sc_finish_round<SC_PRODUCT, T, T>(w, io, k, static_cast<TrWarp&>(tr));
            to_words(rn, r_sh[k & 1]);
        } else if (paired && warp == 1) {
            tr_pair_help(trbuf);
        } else if (role.index >= 0) {
            if (first) pipe_worker_pass(rf, rg, wf, wg, n, false, r, cw, csum[k & 1], role);
            else       pipe_worker_pass(rf, rg, wf, wg, 2 * n, true, r, cw, csum[k & 1], role);
        }
        __syncthreads();
        if (!first) { rf = wf; rg = wg; }            // the fold above wrote dst
        first = false;
        from_words(r, r_sh[k & 1]);                  // r_k
        if (n == 2) break;                           // round k was the last one
        if (warp == 0) {                             // three lanes evaluate the three quadratics, all collect
            if (threadIdx.x < 3) {
                const u32* c = csum[k & 1] + 3 * W * threadIdx.x;
                T c0, c1, c2;
                from_words(c0, c); from_words(c1, c + W); from_words(c2, c + 2 * W);
                to_words(c0 + r * (c1 + r * c2), w_sh + W * threadIdx.x);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 3 * W; i++) w[i] = w_sh[i];
            __syncwarp();
        }
        k++;
        n /= 2;
    }
    (void)num_vars;

    sc_post_squeezes(tr, io, trbuf);
    if (threadIdx.x == 0) {
        tr_store(tr, io.tr);
        // two elements per table remain (folded through r_(k-1)): fold the last challenge in
        T fv = lerp(ld_fe(rf), ld_fe(rf + 1), r), gv = lerp(ld_fe(rg), ld_fe(rg + 1), r);
        to_words(fv, io.fin);
        to_words(gv, io.fin + W);
    }
    ZKB_STAMP_END(io.tr, 1);
}

}  // namespace zkb
