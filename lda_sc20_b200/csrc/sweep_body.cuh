// sweep_body.cuh -- per-unit bodies of the sweep kernels (one word tile, one word, one
// doc, one sampler tile), shared by the single-corpus kernels and the batched ones.
//
// Every float operation below is an explicit round-to-nearest intrinsic, so the compiler
// cannot contract or reorder it.  The sampling arithmetic (summation orders, bin order,
// tie rules) is the specification the CPU oracle restates; the CUDA path and the oracle
// therefore draw identical topics for identical (seed, iteration, token).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "thread_search.cuh"

namespace lda {
namespace dev {

// ---------------------------------------------------------------- WT rebuild
// Warp per word tile: the tile's topics are histogrammed in a warp-private shared row
// with one shared atomic per token (aggregating a warp's equal topics with
// __match_any_sync first made the rebuild 2.6x slower).  Dense tiles add their row into the dense
// word-topic matrix; a sparse word (one tile over all chunks) is compacted to
// (k<<16 | count) ascending k.  Topic totals n_k are privatised per CTA and flushed once.
// Replaces WTDen_Update_Kernel, WT_Update_Kernel, sparseMatrixAdd and
// WTDen_Sum_Update_Kernel (EZLDA/utility.cu:1067-1102, :10-76, :1132-1204, :1104-1126).
struct WtArgs {
    const int4* tiles;  // {word, start, count, dense}
    int ntiles;
    unsigned* tile_counter;
    const uint16_t* z;
    int K, V, Vd, C;
    const uint32_t* seg_off;  // [C*V]
    const uint32_t* seg_cnt;  // [C*V]
    int* dwt;                 // [Vd*K]
    const uint32_t* swt_off;  // [V-Vd]
    uint32_t* swt_nnz;
    uint32_t* swt_ent;
    int* n_k;
    int* err;
};

// One word tile: histogram its topics in the warp's shared row `hist` (K words) with the
// bitmap of its non-zero topics in `bits` (ceil(K/32) words), both zero on entry and on
// exit, and add it to the dense row or write the sparse row (ascending k, placed by a
// prefix scan of the bitmap words' popcounts); topic totals go to `nk` (a CTA-private
// shared array, or the model's global totals).
__device__ __forceinline__ int wt_bit_words(int K) { return (K + 31) >> 5; }

template <class H>
__device__ __forceinline__ void wt_tile(const WtArgs& a, const int4 t, const H& hist, uint32_t* bits, unsigned* nk,
                                        int lane) {
    const int w = t.x;
    if (t.w & 1) {
        hist_segment(a.z, (uint32_t)t.y, (uint32_t)t.z, hist, bits, a.K, lane, a.err);
    } else {
        // a sparse word's segments in every chunk: lane c loads chunk c's offset and count
        for (int c0 = 0; c0 < a.C; c0 += 32) {
            const int c = c0 + lane;
            uint32_t so = 0, sc = 0;
            if (c < a.C) {
                const size_t idx = (size_t)c * a.V + w;
                so = __ldg(a.seg_off + idx);
                sc = __ldg(a.seg_cnt + idx);
            }
            const int nc = min(32, a.C - c0);
            for (int j = 0; j < nc; ++j) {
                const uint32_t o = __shfl_sync(FULL, so, j), n = __shfl_sync(FULL, sc, j);
                if (n) hist_segment(a.z, o, n, hist, bits, a.K, lane, a.err);
            }
        }
    }
    __syncwarp();
    const int words = wt_bit_words(a.K);
    if (t.w & 1) {
        int* row = a.dwt + (size_t)w * a.K;
        for (int wi = lane; wi < words; wi += 32) {
            uint32_t m = bits[wi];
            if (m) bits[wi] = 0u;
            while (m) {
                const uint32_t k = (uint32_t)wi * 32u + (uint32_t)(__ffs(m) - 1);
                m &= m - 1u;
                const uint32_t h = hist.get(k);
                atomicAdd(row + k, (int)h);
                atomicAdd(nk + k, h);
                hist.clear(k);
            }
        }
    } else {
        const int s = w - a.Vd;
        uint32_t* out = a.swt_ent + a.swt_off[s];
        uint32_t nnz = 0;
        for (int wb = 0; wb < words; wb += 32) {
            const int wi = wb + lane;
            uint32_t m = wi < words ? bits[wi] : 0u;
            const uint32_t c = (uint32_t)__popc(m);
            uint32_t incl = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t v = __shfl_up_sync(FULL, incl, off);
                if (lane >= off) incl += v;
            }
            uint32_t p = nnz + incl - c;
            nnz += __shfl_sync(FULL, incl, 31);
            if (m) bits[wi] = 0u;
            while (m) {
                const uint32_t k = (uint32_t)wi * 32u + (uint32_t)(__ffs(m) - 1);
                m &= m - 1u;
                const uint32_t h = hist.get(k);
                out[p++] = (k << 16) | h;
                atomicAdd(nk + k, h);
                hist.clear(k);
            }
        }
        if (lane == 0) a.swt_nnz[s] = nnz;
    }
    __syncwarp();
}

// ---------------------------------------------------------------- word stats
// Warp per word: max / 2nd / 3rd topic of phi (ties to the lower k), phi at those
// topics, and the 32 lane partials of Q = alpha * sum_{k != max} phi_k.  Replaces
// MaxTopicDense_Update_Kernel / MaxTopicSparse_Update_Kernel (EZLDA/utility.cu:305-1062).
struct StatsArgs {
    int V, Vd, K;
    float alpha, beta, Vbeta;
    const int* n_k;
    const int* dwt;
    const uint32_t* swt_off;
    const uint32_t* swt_nnz;
    const uint32_t* swt_ent;
    uint32_t* st_top2;  // (k2 << 16) | maxK
    uint32_t* st_k3;
    float4* st_phi;     // {phi_max, phi_2nd, phi_3rd, Q}
    float* st_ql;       // [V*32]
    const float* smooth = nullptr;  // K > kLargeK: the smoothing table (k_smooth_table)
    int wlo = 0;                    // the words [wlo, V) get statistics (a word range)
    const float* recip = nullptr;   // r_k = 1 / ((float)n_k + V*beta) (k_recip_order)
    const int* order = nullptr;     // the sparse words' topic order (k_recip_order)
    // K > kLargeK: the dense words' Q-round tables (32 lane slots x qrounds float2 per word,
    // read by k_sample_dense_large), or null
    float2* qtab = nullptr;
    int qrounds = 0;
};

// Topics of the order list: the first kOrderList by (beta * r_k desc, k asc).
constexpr int kOrderList = 64;

// (v, k) ranks above (a, i): larger value, ties to the lower topic.
__device__ __forceinline__ bool ranks_above(float v, int k, float a, int i) { return v > a || (v == a && k < i); }

// The reciprocals r_k = 1 / ((float)n_k + V*beta) of a CTA's 32 topics from k0 on, up to
// kLargeK topics beta * r_k in the sampler's column layout (base, else null), and the order of
// the topics outside a word: the first kOrderList by (beta * r_k desc, k asc).  A topic's
// place in the order is the number of topics that rank above it, counted by the CTA's 8
// warps against an eighth of all K each, so K^2 comparisons spread over ceil(K/32) CTAs.
// (64 arg-max rounds of one CTA over the table took 239 us at K=10,000; one CTA per model of a
// batch for all of its K^2 comparisons 200 us at K=2048, now 8.5.)  smf: K floats.
constexpr int kRecipThreads = 256;
__device__ __forceinline__ void recip_order(const int* __restrict__ n_k, int K, float Vbeta, float beta, float* recip,
                                            float* base, int* order, int k0, float* smf) {
    __shared__ int above[32];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < K; k += blockDim.x)
        smf[k] = fmul(beta, __fdiv_rn(1.0f, fadd(__int2float_rn(__ldg(n_k + k)), Vbeta)));
    if (threadIdx.x < 32) above[threadIdx.x] = 0;
    __syncthreads();
    const int k = k0 + lane;
    const float v = k < K ? smf[k] : 0.0f;
    if (wid == 0 && k < K) {
        recip[k] = __fdiv_rn(1.0f, fadd(__int2float_rn(__ldg(n_k + k)), Vbeta));
        if (base) base[col_skew(k)] = v;
    }
    // the CTA's own topics lie in [k0, k0 + 32): before them a topic ranks above with an equal
    // value, after them only with a larger one
    const int part = (((K + 7) >> 3) + 3) & ~3, j0 = min(K, wid * part), j1 = min(K, j0 + part);
    const int k1 = min(K, k0 + 32);
    int n = 0;
    for (int j = max(j0, k0); j < min(j1, k1); ++j) n += ranks_above(smf[j], j, v, k) ? 1 : 0;
    const int a1 = min(j1, k0), b0 = max(j0, k1);
    for (int j = j0; j + 4 <= a1; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(smf + j);
        n += (x.x >= v) + (x.y >= v) + (x.z >= v) + (x.w >= v);
    }
    if (a1 > j0)
        for (int j = j0 + ((a1 - j0) & ~3); j < a1; ++j) n += smf[j] >= v;
    int j = b0;
    for (; j < j1 && (j & 3); ++j) n += smf[j] > v;
    for (; j + 4 <= j1; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(smf + j);
        n += (x.x > v) + (x.y > v) + (x.z > v) + (x.w > v);
    }
    for (; j < j1; ++j) n += smf[j] > v;
    atomicAdd(&above[lane], n);
    __syncthreads();
    if (wid == 0 && k < K && above[lane] < kOrderList) order[above[lane]] = k;
}

__device__ __forceinline__ void top3_insert(float v, int k, float& a1, int& i1, float& a2, int& i2, float& a3, int& i3) {
    if (ranks_above(v, k, a1, i1)) {
        a3 = a2; i3 = i2;
        a2 = a1; i2 = i1;
        a1 = v; i1 = k;
    } else if (ranks_above(v, k, a2, i2)) {
        a3 = a2; i3 = i2;
        a2 = v; i2 = k;
    } else if (ranks_above(v, k, a3, i3)) {
        a3 = v; i3 = k;
    }
}

// The warp's top three from its lanes' (value desc, topic asc) lists.  Values are -1 (an
// empty place) or non-negative, so their bits order like signed integers.
__device__ __forceinline__ void warp_top3(float a1, int i1, float a2, int i2, float a3, int i3, float (&v)[3],
                                          int (&kk)[3]) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const int best = __reduce_max_sync(FULL, __float_as_int(a1));
        const int bk = __reduce_min_sync(FULL, __float_as_int(a1) == best ? i1 : 0x7fffffff);
        v[q] = __int_as_float(best);
        kk[q] = bk;
        if (i1 == bk) {
            a1 = a2; i1 = i2;
            a2 = a3; i2 = i3;
            a3 = -1.0f; i3 = 0x7fffffff;
        }
    }
}

// The first three topics of the order list that a sparse word (bitmap `bits`) lacks, into
// lane 0's top three; if the list runs out, every topic outside the word into the lanes'.
__device__ __forceinline__ void top3_outside(const StatsArgs& a, const int* order, const uint32_t* bits, float& a1,
                                             int& i1, float& a2, int& i2, float& a3, int& i3, int lane) {
    const int L = min(kOrderList, a.K);
    int found = 0, o0 = 0, o1 = 0, o2 = 0;
    for (int b = 0; b < L && found < 3; b += 32) {
        const int j = b + lane;
        const int kj = j < L ? order[j] : 0;
        const bool out = j < L && !((bits[kj >> 5] >> (kj & 31)) & 1u);
        for (unsigned m = __ballot_sync(FULL, out); m && found < 3; m &= m - 1u) {
            const int k = __shfl_sync(FULL, kj, __ffs(m) - 1);
            if (found == 0) o0 = k;
            else if (found == 1) o1 = k;
            else o2 = k;
            ++found;
        }
    }
    if (found == 3) {
        if (lane == 0) {
            top3_insert(fmul(a.beta, __ldg(a.recip + o0)), o0, a1, i1, a2, i2, a3, i3);
            top3_insert(fmul(a.beta, __ldg(a.recip + o1)), o1, a1, i1, a2, i2, a3, i3);
            top3_insert(fmul(a.beta, __ldg(a.recip + o2)), o2, a1, i1, a2, i2, a3, i3);
        }
    } else {
        for (int k = lane; k < a.K; k += 32)
            if (!((bits[k >> 5] >> (k & 31)) & 1u))
                top3_insert(fmul(a.beta, __ldg(a.recip + k)), k, a1, i1, a2, i2, a3, i3);
    }
}

// The statistics of word w from its column of phi: top three, the lane partials of Q (the
// max topic excluded) and Q.
__device__ __forceinline__ void word_stats_column(const StatsArgs& a, int w, const float* col, int lane) {
    // the lane's top three by (phi desc, k asc) in one pass (k ascends, so a strictly larger
    // value is needed to displace), then three warp-wide pops of the lanes' heads
    float a1 = -1.0f, a2 = -1.0f, a3 = -1.0f;
    int i1 = 0x7fffffff, i2 = 0x7fffffff, i3 = 0x7fffffff;
    for (int k = lane; k < a.K; k += 32) {
        const float x = col[k];
        if (x > a1) {
            a3 = a2; i3 = i2;
            a2 = a1; i2 = i1;
            a1 = x; i1 = k;
        } else if (x > a2) {
            a3 = a2; i3 = i2;
            a2 = x; i2 = k;
        } else if (x > a3) {
            a3 = x; i3 = k;
        }
    }
    float v[3];
    int kk[3];
    warp_top3(a1, i1, a2, i2, a3, i3, v, kk);
    const float v1 = v[0], v2 = v[1], v3 = v[2];
    const int k1 = kk[0], k2 = kk[1], k3 = kk[2];
    float ql = 0.0f;
    for (int k = lane; k < a.K; k += 32) if (k != k1) ql = ffma(a.alpha, col[k], ql);
    const float qp = warp_ks_scan(ql, lane);
    const float Q = __shfl_sync(FULL, qp, 31);
    a.st_ql[(size_t)w * 32 + lane] = ql;
    if (lane == 0) {
        a.st_top2[w] = ((uint32_t)k2 << 16) | (uint32_t)k1;
        a.st_k3[w] = (uint32_t)k3;
        a.st_phi[w] = make_float4(v1, v2, v3, Q);
    }
    __syncwarp();
}

// Whether a sparse word of nnz topics puts the base values back into a column kept for the next
// sparse word: up to an eighth of the topics (a sixteenth and a quarter measure the same, in the
// statistics and in the samplers, K=64 to 1500).
__device__ __forceinline__ bool put_back(uint32_t nnz, int K) { return nnz <= (uint32_t)K >> 3; }

// Words of shared memory a warp of the K <= kLargeK statistics uses: a word column (plain
// layout) and a topic bitmap, a multiple of 4.
__host__ __device__ __forceinline__ int stats_warp_words(int K) { return ((K + 3) & ~3) + ((((K + 31) >> 5) + 3) & ~3); }

// Statistics of word w, K <= kLargeK; `col` and `bits` are the warp's (stats_warp_words).
// phi_k = ((float)n_wk + beta) * r_k; EZLDA builds the same column as WTHead
// (utility.cu:1257-1269 sparse, :1698-1702 dense).  A sparse word needs no pass over K
// topics for its top three (its own topics, and the first three of the order list outside
// it) and no column of its own: `col` keeps the column of a word without tokens while
// `clean`, gets the word's topics written over it for the serial Q sums and put back after.
// What is left per topic is one shared load and one fmaf (42 instructions before: 1,357 per
// word at K=1024).
//
// Words without tokens all have the same statistics: a warp keeps the ones it forms first
// (`none`; one corpus and sweep).
struct NoTokenStats {
    bool have = false;
    uint32_t top2 = 0, k3 = 0;
    float4 phi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float ql = 0.0f;
};
__device__ __forceinline__ void word_stats_word(const StatsArgs& a, int w, float* col, uint32_t* bits, bool& clean,
                                                NoTokenStats& none, int lane) {
    const int K = a.K;
    if (w < a.Vd) {
        const int* row = a.dwt + (size_t)w * K;
        for (int k = lane; k < K; k += 32)
            col[k] = fmul(fadd(__int2float_rn(__ldg(row + k)), a.beta), __ldg(a.recip + k));
        __syncwarp();
        word_stats_column(a, w, col, lane);
        clean = false;
        return;
    }
    const uint32_t* ent = a.swt_ent + __ldg(a.swt_off + (w - a.Vd));
    const uint32_t nnz = __ldg(a.swt_nnz + (w - a.Vd));
    if (nnz == 0u && none.have) {
        a.st_ql[(size_t)w * 32 + lane] = none.ql;
        if (lane == 0) {
            a.st_top2[w] = none.top2;
            a.st_k3[w] = none.k3;
            a.st_phi[w] = none.phi;
        }
        return;
    }
    if (!clean) {
        for (int k = lane; k < K; k += 32) col[k] = fmul(a.beta, __ldg(a.recip + k));
        for (int i = lane; i < (K + 31) >> 5; i += 32) bits[i] = 0u;
        __syncwarp();
    }
    float a1 = -1.0f, a2 = -1.0f, a3 = -1.0f;
    int i1 = 0x7fffffff, i2 = 0x7fffffff, i3 = 0x7fffffff;
    for (uint32_t e = lane; e < nnz; e += 32) {
        const uint32_t en = __ldg(ent + e);
        const int k = (int)(en >> 16);
        const float x = fmul(fadd(u2f(en & 0xffffu), a.beta), __ldg(a.recip + k));
        atomicOr(&bits[k >> 5], 1u << (k & 31));
        col[k] = x;
        top3_insert(x, k, a1, i1, a2, i2, a3, i3);
    }
    __syncwarp();
    top3_outside(a, a.order, bits, a1, i1, a2, i2, a3, i3, lane);
    float v[3];
    int kk[3];
    warp_top3(a1, i1, a2, i2, a3, i3, v, kk);
    const int k1 = kk[0];
    if (lane == 0) col[k1] = 0.0f;  // fmaf(alpha, 0, q) is q: the max topic adds nothing
    __syncwarp();
    float ql = 0.0f;
#pragma unroll 8
    for (int k = lane; k < K; k += 32) ql = ffma(a.alpha, col[k], ql);
    const float Q = __shfl_sync(FULL, warp_ks_scan(ql, lane), 31);
    const uint32_t top2 = ((uint32_t)kk[1] << 16) | (uint32_t)k1;
    const float4 ph = make_float4(v[0], v[1], v[2], Q);
    a.st_ql[(size_t)w * 32 + lane] = ql;
    if (lane == 0) {
        a.st_top2[w] = top2;
        a.st_k3[w] = (uint32_t)kk[2];
        a.st_phi[w] = ph;
    }
    if (nnz == 0u) {
        none.have = true;
        none.top2 = top2;
        none.k3 = (uint32_t)kk[2];
        none.phi = ph;
        none.ql = ql;
    }
    __syncwarp();
    clean = put_back(nnz, K);
    if (clean) {
        for (uint32_t e = lane; e < nnz; e += 32) {
            const int k = (int)(__ldg(ent + e) >> 16);
            col[k] = fmul(a.beta, __ldg(a.recip + k));
            bits[k >> 5] = 0u;
        }
        if (lane == 0) col[k1] = fmul(a.beta, __ldg(a.recip + k1));
        __syncwarp();
    }
}

// ---------------------------------------------------------------- DT rebuild
// Warp per doc of one chunk: the doc's topics are gathered through the doc-order ->
// word-sorted map into a warp-private shared histogram, each token's counts of its
// word's max / 2nd topic are scattered to its word-sorted slot, and the histogram is
// compacted to (k<<16 | count) ascending k.  Replaces DT_Update_Kernel
// (EZLDA/utility.cu:79-284).
struct DtArgs {
    uint32_t d_begin, d_end;
    int K;
    const uint32_t* doc_off;    // [D+1] doc-order token offsets
    const uint32_t* dtok_pos;   // [N]
    const uint32_t* dtok_word;  // [N]
    const uint16_t* z;
    const uint32_t* st_top2;
    const uint32_t* dt_off;
    uint32_t* dt_nnz;
    uint32_t* dt_ent;
    uint32_t* meta;             // [N] word-sorted: (n_d,2nd << 16) | n_d,max
    int* err;
    // dtok_pos / dtok_word / meta hold tokens [tok_base, ...) and dt_ent the doc-row
    // entries [dt_base, ...): 0 when the whole corpus is resident, the chunk's first token
    // and first doc-row entry when the chunk is streamed into a slot buffer
    uint32_t tok_base, dt_base;
    // above kLargeK topics: docs of at most small_max tokens are k_dt_build_small's, the
    // rest k_dt_build_cta's (0: all the CTA kernel's)
    uint32_t small_max = 0;
};

// Doc d: its counts in the warp's shared `hist` (K words) and the bitmap of its non-zero
// topics in `bits` (ceil(K/32) words), both zero on entry and on exit; the per-token
// metadata; and the row, compacted from the bitmap: each lane takes 32 topics' bits, an
// exclusive scan of their popcounts places its entries, ascending k.
__device__ __forceinline__ int dt_bit_words(int K) { return (K + 31) >> 5; }

template <class H>
__device__ __forceinline__ void dt_doc(const DtArgs& a, uint32_t d, const H& hist, uint32_t* bits, int lane) {
    const uint32_t b = __ldg(a.doc_off + d), n = __ldg(a.doc_off + d + 1) - b;
    const uint32_t* dpos = a.dtok_pos + (b - a.tok_base);
    const uint32_t* dword = a.dtok_word + (b - a.tok_base);
    // four 32-token steps per pass: their index loads, then their topic gathers, are in
    // flight together
    for (uint32_t base = 0; base < n; base += 128) {
        uint32_t k[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t i = base + 32u * s + lane;
            k[s] = i < n ? __ldg(dpos + i) : 0xffffffffu;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) k[s] = k[s] != 0xffffffffu ? (uint32_t)__ldg(a.z + k[s]) : 0xffffffffu;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            bool valid = k[s] != 0xffffffffu;
            uint32_t kk = k[s];
            if (valid && kk >= (uint32_t)a.K) {
                atomicOr(a.err, 1);
                valid = false;
                kk = 0xfffffffeu;
            }
            if (valid) hist_token(hist, bits, kk);
        }
    }
    __syncwarp();
    for (uint32_t base = 0; base < n; base += 128) {
        uint32_t pos[4], t2[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t i = base + 32u * s + lane;
            pos[s] = i < n ? __ldg(dpos + i) : 0xffffffffu;
            t2[s] = i < n ? __ldg(dword + i) : 0u;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) t2[s] = pos[s] != 0xffffffffu ? __ldg(a.st_top2 + t2[s]) : 0u;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (pos[s] == 0xffffffffu) continue;
            const uint32_t k1 = t2[s] & 0xffffu, k2 = t2[s] >> 16;
            const uint32_t c1 = k1 < (uint32_t)a.K ? hist.get(k1) : 0u, c2 = k2 < (uint32_t)a.K ? hist.get(k2) : 0u;
            a.meta[pos[s] - a.tok_base] = (c2 << 16) | c1;
        }
    }
    __syncwarp();
    uint32_t* out = a.dt_ent + (__ldg(a.dt_off + d) - a.dt_base);
    const int words = dt_bit_words(a.K);
    uint32_t nnz = 0;
    for (int wb = 0; wb < words; wb += 32) {
        const int wi = wb + lane;
        uint32_t m = wi < words ? bits[wi] : 0u;
        const uint32_t c = (uint32_t)__popc(m);
        uint32_t incl = c;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, incl, off);
            if (lane >= off) incl += t;
        }
        uint32_t p = nnz + incl - c;
        nnz += __shfl_sync(FULL, incl, 31);
        if (m) bits[wi] = 0u;
        while (m) {
            const uint32_t k = (uint32_t)wi * 32u + (uint32_t)(__ffs(m) - 1);
            m &= m - 1u;
            out[p++] = (row_key(a.K, k) << 16) | hist.get(k);
            hist.clear(k);
        }
    }
    if (lane == 0) a.dt_nnz[d] = nnz;
    __syncwarp();
}

// ------------------------------------------------------------------- sampler
// Warp per (word, token range) tile.  The word's phi column (phi_max zeroed) sits in
// warp-private shared memory.  Each 32-token group is screened thread-per-token by the
// max-topic bound; the tokens the bound does not settle (all tokens in LL mode) then need
//   S      lane l's sum over the doc row's entries l, l+32, l+64, ... (coalesced loads, the
//          whole warp per row), a Kogge-Stone scan of the 32 lane sums; a row is summed once
//          for consecutive tokens of the same (word, doc) in the tile;
//   bucket the first lane prefix above the target picks the lane of an S-bucket draw, then
//          a draw among its (at most ceil(nnz/32)) entries; scans, searches and draws run
//          thread-per-token, all the group's tokens at once (sample_groups);
//   Q      a lane by the per-word lane prefixes of Q, then one of its topics k = l, l+32, ...
//          (32 per round, carried).
// Replaces UpdateProbKernelTrainD1, LDAKernelTrainD and LDAKernelTrain
// (EZLDA/utility.cu:2680-3312, :1625-2103, :1217-1611) in one pass, with no
// effective-token list in global memory and no spin lock.
struct SampleArgs {
    const int4* tiles;  // {word, start, count, dense}
    int ntiles;
    unsigned* tile_counter;
    double* tile_ll;
    int K, Vd, ll_mode;
    float alpha, beta;
    double den_add;  // (double)K * (double)alpha
    uint32_t seed_lo, seed_hi, iter;
    const int* dwt;
    const uint32_t* swt_off;
    const uint32_t* swt_nnz;
    const uint32_t* swt_ent;
    const uint32_t* st_top2;
    const float4* st_phi;
    const float* st_ql;
    const uint32_t* tok_doc;
    const uint32_t* meta;
    uint16_t* z;
    const uint32_t* doc_len;
    const uint32_t* dt_off;
    const uint32_t* dt_nnz;
    const uint32_t* dt_ent;
    // tokens, ea, full, sum_nnz, max, s, q, word_nnz, dense tiles, sparse tiles, rows, row entries
    unsigned long long* ctr;
    // tok_doc / meta hold tokens [tok_base, ...) and dt_ent the doc-row entries
    // [dt_base, ...) (non-zero when the chunk is streamed into a slot buffer)
    uint32_t tok_base, dt_base;
    // r_k = 1 / ((float)n_k + V*beta) for k < K, formed once per sweep or call (per column
    // instead, an allocation-free call at K=12,000 took 1,334 us against 627)
    const float* recip = nullptr;
    // K <= kLargeK: beta * r_k in the skewed column layout, the column of a word without
    // tokens (col_words(K) floats, formed with recip)
    const float* base = nullptr;
    int nslots = 1;  // row slots per warp (sample_groups)
    // K > kLargeK: the smoothing table of the split Q bucket (k_smooth_table)
    const float* smooth = nullptr;
    // K > kLargeK: the dense words' Q-round tables (k_word_stats_dense_cta), or null
    const float2* qtab_g = nullptr;
};

// The split Q bucket of a sparse word above kLargeK topics: Q = Qw + Qs, Qw over the word's
// own topics, Qs the word-independent smoothing part alpha * beta * sum_{k != max} r_k.
struct SplitQ {
    const uint32_t* ent;  // the word's row (k << 16 | count), ascending k
    uint32_t nnz;
    float Qw;
    const float* T;       // the smoothing table (K entries, ascending but for rounding)
    const float* r;       // r_k
    // the Qw rounds' table, lane r holding round r's (carry before it, carry + its largest
    // KS prefix); rounds = 0 when not built (more than 32 rounds, or not wanted)
    int rounds = 0;
    float qcarry = 0.0f, qthr = 0.0f;
    // in shared memory, for thread_split_draw: the prefixes of a one-round word's terms (else
    // null) with the entries whose term is positive, and the last entry of each of T's rounds
    const float* wp = nullptr;
    unsigned wok = 0u;
    const float* tend = nullptr;
    __device__ __forceinline__ float rk(int k) const { return __ldg(r + k); }
    // round slot i of the Qw search: alpha * (n_wk * r_k), the max topic's term 0
    __device__ __forceinline__ void slot(uint32_t i, int maxK, float alpha, int& key, float& term, bool& ok) const {
        const uint32_t en = __ldg(ent + i);
        const int k = (int)(en >> 16);
        term = k == maxK ? 0.0f : fmul(alpha, fmul(u2f(en & 0xffffu), rk(k)));
        key = k;
        ok = term > 0.0f;
    }
};

// Builds the Qw rounds' table of a split word (2 to 32 rounds of 32 entries): each
// round's total and largest lane prefix from its Kogge-Stone scan, and the carries as the
// fadd chain of the totals, the values warp_level2 forms round by round.  Warp-uniform.
__device__ __forceinline__ void split_q_table(SplitQ& q, int maxK, float alpha, int lane) {
    const uint32_t R = (q.nnz + 31u) >> 5;
    if (R < 2 || R > 32) return;  // one round: the walk is that round already
    float carry = 0.0f;
    for (uint32_t r = 0; r < R; ++r) {
        int key = -1;
        float term = 0.0f;
        bool ok = false;
        const uint32_t i = 32u * r + (uint32_t)lane;
        if (i < q.nnz) q.slot(i, maxK, alpha, key, term, ok);
        const float ks = warp_ks_scan(term, lane);
        float mx = ks;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, off));
        const float tot = __shfl_sync(FULL, ks, 31);
        if ((uint32_t)lane == r) {
            q.qcarry = carry;
            q.qthr = fadd(carry, mx);
        }
        carry = fadd(carry, tot);
    }
    q.rounds = (int)R;
}

// The Q-bucket draw of a split word for t = target - pS (uniform across the warp): the
// word's own topics first, in rounds of 32 entries (carry + Kogge-Stone scan of
// alpha * (n_wk * r_k), the max topic's term 0; the first entry with a non-zero term whose
// prefix exceeds t, else the last such entry); otherwise smoothing for t' = t - Qw against
// T with the max topic left out: the first k < maxK with t' < T[k] when t' < T[maxK-1],
// else the first k > maxK with t' + sm_max < T[k], else the last topic other than maxK.
__device__ __forceinline__ int split_q_draw(const SplitQ& q, float t, int maxK, int K, float alpha, float beta,
                                            int lane) {
    if (t < q.Qw) {
        auto slot = [&](uint32_t i, int& key, float& term, bool& ok) { q.slot(i, maxK, alpha, key, term, ok); };
        int z = -1;
        if (q.rounds > 0) {
            // the candidate rounds (t below the round's largest prefix), in order
            for (unsigned b = __ballot_sync(FULL, lane < q.rounds && t < q.qthr); b; b &= b - 1u) {
                const uint32_t r = (uint32_t)(__ffs(b) - 1);
                const float carry = __shfl_sync(FULL, q.qcarry, (int)r);
                int key = -1;
                float term = 0.0f;
                bool ok = false;
                const uint32_t i = 32u * r + (uint32_t)lane;
                if (i < q.nnz) slot(i, key, term, ok);
                const float ks = warp_ks_scan(term, lane);
                const unsigned f = __ballot_sync(FULL, ok && t < fadd(carry, ks));
                if (f) {
                    z = __shfl_sync(FULL, key, __ffs(f) - 1);
                    break;
                }
            }
        }
        if (z < 0) z = warp_level2(q.nnz, t, -1, lane, slot);
        if (z >= 0) return z;
    }
    const float t1 = fsub(t, q.Qw);
    if (maxK > 0 && t1 < __ldg(q.T + maxK - 1)) return warp_first_above(q.T, 0, maxK, t1, lane);
    const float t2 = fadd(t1, fmul(alpha, fmul(beta, q.rk(maxK))));
    const int z = warp_first_above(q.T, maxK + 1, K, t2, lane);
    return z >= 0 ? z : (maxK == K - 1 ? K - 2 : K - 1);
}



// Sweep counters live in shared memory (one row per warp, written by lane 0) so they
// cost no registers in the sampling loop.
enum { C_TOK, C_EA, C_FULL, C_NNZ, C_MAX, C_S, C_Q, C_WNNZ, C_TDENSE, C_TSPARSE, C_ROWS, C_RENT, C_NUM };

// Warps per CTA of the K <= 2048 sampler (one shared word column per warp), and the CTAs
// per SM it is compiled for: the register cap is 65536 / (32 * warps * blocks) per
// thread.  A thread holds a row's 32 lane sums, so the plain kernels take 4 CTAs (64
// registers; 5 CTAs of 48 spill: 1.96 against 1.92 ms per sweep at K=1024, and 3 leave too
// few warps, 2.23 ms).  The K > 1024 kernels (several Q rounds per batch) and the LL kernel up
// to kThreadQTopics (its FP64 products; K=64: 119 -> 109 us per sweep) take 3; above, the LL
// kernel spills 44 bytes at 4 and is still faster (K=1024: 701 against 755 us).

#ifndef LDA_SAMPLE_WARPS
#define LDA_SAMPLE_WARPS 8
#endif
constexpr int kSampleWarps = LDA_SAMPLE_WARPS;
#ifndef LDA_SAMPLE_MIN_BLOCKS
#define LDA_SAMPLE_MIN_BLOCKS 4
#endif
#ifndef LDA_SAMPLE_QB_MIN_BLOCKS
#define LDA_SAMPLE_QB_MIN_BLOCKS 3
#endif
#ifndef LDA_SAMPLE_LL_MIN_BLOCKS
#define LDA_SAMPLE_LL_MIN_BLOCKS 4
#endif
constexpr int kSampleLL0MinBlocks = 3;

// The slots in which a warp keeps doc rows' lane sums: row slot s holds the 32 sums of one
// row at [33 s, 33 s + 32), so that 32 threads reading element i of 32 different rows touch
// 32 banks.
constexpr int kSlotWords = 33;
// Words of a warp's row slots, even (the rows' list, 32 x {offset, length}, follows them).
__host__ __device__ __forceinline__ int slot_words(int nslots) { return (kSlotWords * nslots + 1) & ~1; }
__host__ __device__ __forceinline__ int row_state_words(int nslots) { return slot_words(nslots) + 64; }

// The branch that a token's draw takes: early accepts and tokens without a draw have none.
enum { BR_NONE = 0, BR_MAX = 1, BR_S = 2, BR_Q = 3 };

// What a group's tokens drew so far: the branch, and for the S bucket the lane and the rest
// of the target inside it, for the Q bucket the rest of the target.
struct Draw {
    int kind;
    uint32_t ls;
    float t;
    float total;  // LL mode: S + Q + the max topic's term
};

// Fewest tokens that decide_tokens takes thread per token: below, the whole warp decides
// them one by one (about 45 warp instructions each against 280; from 7 tokens on instead, 1.96
// against 1.92 ms per sweep at K=1024).
constexpr int kDecideMin = 3;

// The tokens (lane = token, those with `act`) whose doc row's lane sums sit in slot my_s of
// `slots`: S from the row's 32 sums, the branch, and for an S-bucket draw the lane: the
// first whose prefix exceeds the target and whose sum is positive, else the last with a
// positive sum.  Thread per token, each scanning its row's sums in registers and searching
// the prefixes; a token whose search is not sure, and all of a few tokens, are decided by
// the whole warp.
template <bool LL>
__device__ __forceinline__ void decide_tokens(const float* slots, int my_s, bool act, bool ea, float pmax, float Q,
                                              float u, int lane, Draw& dr) {
    unsigned by_warp = __ballot_sync(FULL, act);
    if (__popc(by_warp) >= kDecideMin) {
        const float* p = slots + kSlotWords * my_s;
        float v[32];
#pragma unroll
        for (int l = 0; l < 32; ++l) v[l] = p[l];
        thread_ks_scan(v);
        const float pS = fadd(pmax, v[31]);
        const float total = fadd(pS, Q);
        const float target = fmul(u, total);
        const float tt = fsub(target, pmax);
        int ls;
        float prev;
        bool sure;
        thread_crossing(v, tt, ls, prev, sure);
        bool slow = false;
        if (act) {
            if (LL) dr.total = total;
            if (!LL || !ea) {
                if (target < pmax) {
                    dr.kind = BR_MAX;
                } else if (target < pS) {
                    dr.kind = BR_S;
                    dr.ls = (uint32_t)ls;
                    dr.t = ls > 0 ? fsub(tt, prev) : tt;
                    slow = !sure || !(p[ls] > 0.0f);
                } else {
                    dr.kind = BR_Q;
                    dr.t = fsub(target, pS);
                }
            }
        }
        by_warp = __ballot_sync(FULL, slow);
    }
    for (; by_warp; by_warp &= by_warp - 1u) {
        const int j = __ffs(by_warp) - 1;
        const float SL = slots[kSlotWords * __shfl_sync(FULL, my_s, j) + lane];
        const float SP = warp_ks_scan(SL, lane);
        const float pmj = __shfl_sync(FULL, pmax, j);
        const float pS = fadd(pmj, __shfl_sync(FULL, SP, 31));
        const float total = fadd(pS, __shfl_sync(FULL, Q, j));
        const float target = fmul(__shfl_sync(FULL, u, j), total);
        const float tt = fsub(target, pmj);
        const unsigned cand = __ballot_sync(FULL, tt < SP && SL > 0.0f), pos = __ballot_sync(FULL, SL > 0.0f);
        const int ls = cand ? __ffs(cand) - 1 : 31 - __clz(pos);
        const float prev = __shfl_sync(FULL, SP, ls > 0 ? ls - 1 : 0);
        if (lane == j) {
            if (LL) dr.total = total;
            if (!LL || !ea) {
                const bool s = target < pS;
                dr.kind = target < pmj ? BR_MAX : (s ? BR_S : BR_Q);
                dr.ls = (uint32_t)ls;
                dr.t = s ? (ls > 0 ? fsub(tt, prev) : tt) : fsub(target, pS);
            }
        }
    }
}

// A Q-bucket draw of a word by its column, for the rest tt of the target (the whole warp
// works on one token): the lane from the word's Q partials, then one of its topics.
template <int QB, class View>
__device__ __forceinline__ int warp_q_draw(const View& colz, float tt, float QL, float QP, int K, float alpha, int maxK,
                                           int lane, const float2* qtab, int qrounds) {
    const unsigned cand = __ballot_sync(FULL, tt < QP && QL > 0.0f);
    const unsigned pos = __ballot_sync(FULL, QL > 0.0f);
    const int ls = cand ? __ffs(cand) - 1 : (pos ? 31 - __clz(pos) : 0);
    const float prev = __shfl_sync(FULL, QP, ls > 0 ? ls - 1 : 0);
    const float t2 = ls > 0 ? fsub(tt, prev) : tt;
    const uint32_t n = (uint32_t)((K - ls + 31) / 32);
    auto slot = [&](uint32_t i, int& key, float& term, bool& ok) {
        const int k = ls + 32 * (int)i;
        const float cz = colz(k);
        key = k;
        term = fmul(alpha, cz);
        ok = cz > 0.0f;
    };
    int z = qtab ? warp_level2_table(n, t2, lane, slot, qtab + ls * qrounds) : -1;
    if (z < 0) z = warp_level2_rounds<QB>(n, t2, maxK, lane, slot);
    return z;
}

// Above kLargeK, fewest Q-bucket draws of a group that run thread per token (three quarters
// of the draws are from Q there while a model is young: K=10,000, 10M tokens 4.40 ms per
// sweep; from 8 draws on 4.45, none 4.90).
constexpr int kThreadQMin = 4;

// The 32-token groups g0, g0 + gstep, ... of the token range [start, start + cnt) of one
// word (column view colz, max topic maxK, phi4 ph, Q partials QL / QP / Q of the word), or,
// with a shared group counter gq, the groups the warp claims from it (32 tokens at a time,
// so that the warps sharing a tile finish it together).  `slots` holds the warp's a.nslots
// row slots and its list of a group's rows (row_state_words).  Returns the lane's LL partial (LL mode).
//
// A group runs in three parts: its tokens are screened thread-per-token; the doc rows that
// the unsettled tokens need are summed one after another by the whole warp into the slots
// (consecutive tokens of one doc share a row, also across groups); then each token's thread
// scans its row's 32 lane sums, forms S and picks bucket and lane by itself.  Deciding each
// token with the whole warp (a scan by shuffles, ballots and broadcasts per token) took
// about half of the kernel's instructions, and the kernel is bound by their issue.
template <bool LL, int QB, bool SPLIT = false, class View>
__device__ __forceinline__ double sample_groups(const SampleArgs& a, uint32_t start, uint32_t cnt, uint32_t g0,
                                                uint32_t gstep, uint32_t iter, int maxK, const float4 ph, float QL,
                                                float QP, float Q, const View& colz, uint32_t* ctr, int lane,
                                                float* slots, const float2* qtab = nullptr, int qrounds = 0,
                                                const SplitQ* sq = nullptr, uint32_t* gq = nullptr,
                                                float* qps = nullptr) {
    auto claim = [&]() {
        uint32_t v = 0;
        if (lane == 0) v = atomicAdd(gq, 32u);
        return __shfl_sync(FULL, v, 0);
    };
    double ll = 0.0;
    // LL mode: the lane's factors total_t and (n_d + K alpha) as FP64 products, one log of
    // their ratio per 16 tokens (earlier if a product leaves [1e-150, 1e150])
    double ll_num = 1.0, ll_den = 1.0;
    int ll_n = 0;
    using E = typename View::Entry;
    const E* rows = reinterpret_cast<const E*>(a.dt_ent);
    const int nslots = a.nslots;
    uint2* list = reinterpret_cast<uint2*>(slots + slot_words(nslots));
    const unsigned qpos = __ballot_sync(FULL, QL > 0.0f);
    if (QB == 0) {
        qps = reinterpret_cast<float*>(ctr + ((C_NUM + 3) & ~3));  // the word's Q prefixes
        qps[lane] = QP;
        __syncwarp();
    }
    uint32_t cur = 0xffffffffu;  // the doc of the last row summed, in slot cslot
    int cslot = 0;
    for (uint32_t g = gq ? claim() : g0; g < cnt; g = gq ? claim() : g + gstep) {
        const bool valid = g + lane < cnt;
        const uint32_t tok = start + g + lane;
        uint32_t d = 0xffffffffu, nd = 0, my_nnz = 0, my_off = 0;
        float u = 0.0f, pmax = 0.0f;
        bool ea = false;
        if (valid) {
            d = __ldg(a.tok_doc + (tok - a.tok_base));
            const uint32_t m = __ldg(a.meta + (tok - a.tok_base));
            nd = __ldg(a.doc_len + d);
            my_nnz = __ldg(a.dt_nnz + d);
            my_off = __ldg(a.dt_off + d) - a.dt_base;
            const uint32_t cmax = m & 0xffffu, c2 = m >> 16;
            u = token_uniform(a.seed_lo, a.seed_hi, iter, tok);
            pmax = fmul(fadd(u2f(cmax), a.alpha), ph.x);
            const float shat = ffma(u2f(c2), ph.y, fmul(u2f(nd - cmax - c2), ph.z));
            const float bound = fadd(fadd(pmax, shat), Q);
            ea = fmul(u, bound) < pmax;
        }
        int znew = maxK;
        Draw dr{BR_NONE, 0u, 0.0f, 0.0f};
        const unsigned vmask = __ballot_sync(FULL, valid);
        const unsigned emask = __ballot_sync(FULL, ea);
        const unsigned need = LL ? vmask : (vmask & ~emask);
        const bool mine = (need >> lane) & 1u;
        // the tokens that start a new row: those whose doc differs from the previous
        // evaluated token's (the last group's last row for the first)
        const unsigned below = need & ((1u << lane) - 1u);
        uint32_t dp = __shfl_sync(FULL, d, below ? 31 - __clz(below) : lane);
        if (!below) dp = cur;
        const bool lead = mine && d != dp;
        const unsigned leaders = __ballot_sync(FULL, lead);
        if (need) {
            // the group's rows in order: row 0 is the carried one when its first token's doc
            // was the last one summed (its sums move to the first slot); rows r0 + i of a
            // part sit in slot i.  The rows' places and lengths wait in `list`.
            const bool carried = !(leaders & need & (0u - need));
            const int c1 = carried ? 1 : 0;
            const int nrows = __popc(leaders) + c1;
            const int ri = __popc(leaders & ((2u << lane) - 1u)) - 1 + c1;
            if (lead) list[ri] = make_uint2(my_off, my_nnz);
            if (carried) slots[lane] = slots[kSlotWords * cslot + lane];
            __syncwarp();
            for (int r0 = 0; r0 < nrows; r0 += nslots) {
                const int n = min(nrows - r0, nslots);
                float* out = slots + lane;
                int i = 0;
                if (r0 == 0) {
                    i = c1;
                    out += kSlotWords * c1;
                }
                if constexpr (View::kAhead && (!LL || QB == 0)) {
                    // the next row's first steps are loaded while a row is summed (K=1024,
                    // 14.4M tokens: 1.92 -> 1.87 ms per sweep; the LL kernels above
                    // kThreadQTopics spill and lose 1%)
                    uint2 q = make_uint2(0u, 0u);
                    uint32_t e[4] = {}, f[4];
                    if (i < n) {
                        q = list[r0 + i];
                        row_load(e, rows + q.x, (uint32_t)lane, q.y);
                    }
#pragma unroll(QB == 0 ? 2 : 1)
                    for (; i < n; ++i, out += kSlotWords) {
                        const uint2 c = q;
#pragma unroll
                        for (int j = 0; j < 4; ++j) f[j] = e[j];
                        if (i + 1 < n) {
                            q = list[r0 + i + 1];
                            row_load(e, rows + q.x, (uint32_t)lane, q.y);
                        }
                        *out = row_sum(f, rows + c.x, (uint32_t)lane, c.y, colz);
                    }
                } else {
                    for (; i < n; ++i, out += kSlotWords) {
                        const uint2 q = list[r0 + i];
                        if constexpr (SPLIT && View::kOwnMass) *out = colz.mass(rows + q.x, (uint32_t)lane, q.y);
                        else *out = lane_mass(rows + q.x, (uint32_t)lane, q.y, colz);
                    }
                }
                __syncwarp();
                // the tokens of these rows, thread per token
                const bool act = mine && (unsigned)(ri - r0) < (unsigned)n;
                const int my_s = act ? ri - r0 : 0;
                decide_tokens<LL>(slots, my_s, act, ea, pmax, Q, u, lane, dr);
                __syncwarp();  // the slots may be overwritten
            }
            cslot = (nrows - 1) % nslots;
            cur = __shfl_sync(FULL, d, 31 - __clz(need));
        }
        const unsigned qm = __ballot_sync(FULL, dr.kind == BR_Q);
        unsigned by_warp = qm;
        if (QB == 0 && qm) {
            bool unsure;
            const int zq = thread_q_draw(colz, qps, qpos, dr.t, a.K, a.alpha, maxK, unsure);
            if (dr.kind == BR_Q) znew = zq;
            by_warp = __ballot_sync(FULL, dr.kind == BR_Q && unsure);
        }
        if (SPLIT && sq->tend && __popc(qm) >= kThreadQMin) {
            bool unsure = false;
            int zq = maxK;
            if (dr.kind == BR_Q) zq = thread_split_draw(*sq, dr.t, maxK, a.K, a.alpha, a.beta, unsure);
            if (dr.kind == BR_Q) znew = zq;
            by_warp = __ballot_sync(FULL, unsure);
        }
        if (QB > 1 && !SPLIT && qtab && __popc(qm) >= kThreadQMin) {
            bool unsure = false;
            int zq = maxK;
            if (dr.kind == BR_Q) zq = thread_q_draw_table(colz, qps, qpos, dr.t, a.K, a.alpha, qtab, qrounds, unsure);
            if (dr.kind == BR_Q) znew = zq;
            by_warp = __ballot_sync(FULL, unsure);
        }
        for (; by_warp; by_warp &= by_warp - 1u) {
            const int j = __ffs(by_warp) - 1;
            const float tt = __shfl_sync(FULL, dr.t, j);
            int zq;
            if (SPLIT) zq = split_q_draw(*sq, tt, maxK, a.K, a.alpha, a.beta, lane);
            else zq = warp_q_draw<QB == 0 ? 1 : QB>(colz, tt, QL, QP, a.K, a.alpha, maxK, lane, qtab, qrounds);
            if (lane == j) znew = zq;
        }
        // each lane's own token's log-likelihood factors, all lanes at once (every lane
        // accumulates only its own tokens, in group order)
        if (LL && valid) {
            ll_num *= (double)dr.total;
            ll_den *= (double)nd + a.den_add;
            if (++ll_n == 16 || ll_num < 1e-150 || ll_num > 1e150 || ll_den > 1e150) {
                ll += log(ll_num / ll_den);
                ll_num = ll_den = 1.0;
                ll_n = 0;
            }
        }
        // an S-bucket token's row is its own doc's: the lane holds its offset and length
        if (dr.kind == BR_S) znew = lane_draw(rows + my_off, dr.ls, my_nnz, colz, dr.t, maxK);
        if (valid) a.z[tok] = (uint16_t)znew;
        // counters of the group: ballots and warp sums instead of per-token updates
        const unsigned sm = __ballot_sync(FULL, dr.kind == BR_S), xm = __ballot_sync(FULL, dr.kind == BR_MAX);
        const uint32_t nnz_full = __reduce_add_sync(FULL, mine ? my_nnz : 0u);
        const uint32_t nnz_rows = __reduce_add_sync(FULL, lead ? my_nnz : 0u);
        if (lane == 0) {
            ctr[C_TOK] += __popc(vmask);
            ctr[C_EA] += __popc(emask);
            ctr[C_FULL] += __popc(need);
            ctr[C_NNZ] += nnz_full;
            ctr[C_MAX] += __popc(xm) + __popc(emask);
            ctr[C_S] += __popc(sm);
            ctr[C_Q] += __popc(qm);
            ctr[C_ROWS] += __popc(leaders);
            ctr[C_RENT] += nnz_rows;
        }
    }
    if (LL && ll_n) ll += log(ll_num / ll_den);
    return ll;
}

// Words of shared memory that a warp of the column samplers uses: its word column, its row
// slots, its counter row and (QB 0) the word's Q prefixes, a multiple of 4 (the columns are
// 16-byte aligned).
__host__ __device__ __forceinline__ int sample_warp_words(int K, int nslots) {
    return col_words(K) + ((row_state_words(nslots) + 3) & ~3) + ((C_NUM + 3) & ~3) + (K <= kThreadQTopics ? 32 : 0);
}

// One sampler tile (tile index `tile` of a.tiles, content t) with the word column in the
// warp's shared `col` (col_words(K) floats, skewed layout), its row slots and its shared
// counter row `ctr`.  QB: Q-bucket rounds decided per batch (1 for K <= 1024, where a lane
// has one round of topics; 0 for K <= kThreadQTopics).  `held`: the dense word whose column
// `col` holds, or kHoldsBase for the column of a word without tokens (a.base): a sparse
// word's column is that with the word's own topics written over it, and a word with few of
// them puts the base values back when the tile is done, so that the next sparse word costs
// its own entries instead of K, and a dense word's next tile nothing.  (Forming every tile's column
// anew cost 160 warp instructions at K=1024, where an average tile has 31 tokens on a
// corpus of 14M tokens.)  Without a.base the column is formed in full from n_k.
constexpr int kHoldsNone = -1, kHoldsBase = -2;
template <bool LL, int QB = 1, bool SKEWKEYS = true>
__device__ __forceinline__ void sample_tile(const SampleArgs& a, int tile, const int4 t, uint32_t iter, float* col,
                                            float* slots, int& held, uint32_t* ctr, int lane) {
    using View = ColSharedT<SKEWKEYS>;
    const int w = t.x;
    const uint32_t start = (uint32_t)t.y, cnt = (uint32_t)t.z;
    const bool sparse = w >= a.Vd;
    const int maxK = (int)(__ldg(a.st_top2 + w) & 0xffffu);
    const float4 ph = __ldg(a.st_phi + w);
    const float QL = __ldg(a.st_ql + (size_t)w * 32 + lane);
    const uint32_t* ent = a.swt_ent;
    uint32_t nnz = 0;
    if (sparse) {
        ent += __ldg(a.swt_off + (w - a.Vd));
        nnz = __ldg(a.swt_nnz + (w - a.Vd));
    }
    __syncwarp();
    bool clean = false;
    if (!sparse) {
        const int* row = a.dwt + (size_t)w * a.K;
        if (!SKEWKEYS || held != w)
            for (int k = lane; k < a.K; k += 32)
                col[col_skew(k)] = fmul(fadd(__int2float_rn(__ldg(row + k)), a.beta), __ldg(a.recip + k));
        held = w;
    } else {
        if (SKEWKEYS) {
            if (held != kHoldsBase) {
                const float4* src = reinterpret_cast<const float4*>(a.base);
                for (int i = lane; i < col_words(a.K) / 4; i += 32) reinterpret_cast<float4*>(col)[i] = __ldg(src + i);
            }
        } else {
            for (int k = lane; k < a.K; k += 32) col[col_skew(k)] = fmul(a.beta, __ldg(a.recip + k));
        }
        __syncwarp();
        for (uint32_t e = lane; e < nnz; e += 32) {
            const uint32_t en = __ldg(ent + e);
            const int k = (int)(en >> 16);
            col[col_skew(k)] = fmul(fadd(u2f(en & 0xffffu), a.beta), __ldg(a.recip + k));
        }
        clean = SKEWKEYS && put_back(nnz, a.K);
        held = clean ? kHoldsBase : kHoldsNone;
    }
    __syncwarp();
    if (lane == 0) {
        ctr[C_WNNZ] += nnz;
        ctr[sparse ? C_TSPARSE : C_TDENSE] += 1u;
        col[col_skew(maxK)] = 0.0f;
    }
    const float QP = warp_ks_scan(QL, lane);
    const float Q = __shfl_sync(FULL, QP, 31);
    __syncwarp();
    double ll;
    bool split = false;
    if constexpr (QB > 1 && !SKEWKEYS) split = a.K > kLargeK && sparse;
    if (split) {
        // a sparse word above kLargeK topics: the split Q bucket
        if constexpr (QB > 1 && !SKEWKEYS) {
            const SplitQ sq{ent, nnz, __shfl_sync(FULL, QL, 0), a.smooth, a.recip};
            ll = sample_groups<LL, QB, true>(a, start, cnt, 0u, 32u, iter, maxK, ph, QL, QP, Q, View{col}, ctr, lane,
                                             slots, nullptr, 0, &sq);
        }
    } else {
        ll = sample_groups<LL, QB>(a, start, cnt, 0u, 32u, iter, maxK, ph, QL, QP, Q, View{col}, ctr, lane, slots);
    }
    if (LL) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) ll += __shfl_xor_sync(FULL, ll, off);
        if (lane == 0) a.tile_ll[tile] = ll;
    }
    if (clean) {
        __syncwarp();
        for (uint32_t e = lane; e < nnz; e += 32) {
            const int i = col_skew((int)(__ldg(ent + e) >> 16));
            col[i] = __ldg(a.base + i);
        }
        if (lane == 0) col[col_skew(maxK)] = __ldg(a.base + col_skew(maxK));
    }
}

}  // namespace dev
}  // namespace lda
