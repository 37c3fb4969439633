// kernels.cuh -- sm_100a kernels of the collapsed-Gibbs sweep.
//
// Every float operation below is an explicit round-to-nearest intrinsic, so the compiler
// cannot contract or reorder it.  The sampling arithmetic (summation orders, bin order,
// tie rules) is the specification the CPU oracle restates; the CUDA path and the oracle
// therefore draw identical topics for identical (seed, iteration, token).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "sweep_body.cuh"

namespace lda {
namespace dev {

// Tiles are claimed from a counter that stays zero between launches: every claimant (a warp
// or a CTA) makes exactly one claim that finds no tile left, so the claimant that gets
// ntiles + claimants - 1 is the last one of all and puts the counter back.  One thread of
// the claimant calls it with what its claim returned.
__device__ __forceinline__ void last_claim_resets(unsigned* counter, int got, int ntiles, int claimants) {
    if (got == ntiles + claimants - 1) atomicExch(counter, 0u);
}
__device__ __forceinline__ int claim_warp(unsigned* counter, int ntiles, int lane) {
    int tile = 0;
    if (lane == 0) {
        tile = (int)atomicAdd(counter, 1u);
        last_claim_resets(counter, tile, ntiles, (int)(gridDim.x * (blockDim.x >> 5)));
    }
    return tile;  // lane 0's
}

// Zeroes the topic totals and the dense word-topic rows (n4 16-byte pieces of them, then the
// rest) before a rebuild: one launch instead of a memset each.
__global__ void __launch_bounds__(256) k_zero_counts(int* n_k, int K, int4* dwt, int64_t n4, int* rest, int nrest) {
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, st = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = i0; i < n4; i += st) dwt[i] = make_int4(0, 0, 0, 0);
    for (int64_t i = i0; i < K; i += st) n_k[i] = 0;
    if (i0 < nrest) rest[i0] = 0;
}

// Word-topic rebuild: warp per word tile, topic totals privatised per CTA.  P16: 16-bit
// histogram counts (a dense tile holds at most 16,384 tokens and a sparse word fewer than
// 65,536, so every count fits).
template <bool P16>
__global__ void __launch_bounds__(256) k_wt_build(WtArgs a) {
    extern __shared__ uint32_t smu[];
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hw = Hist<P16>::words(a.K);
    const int per = hw + wt_bit_words(a.K);
    uint32_t* nk = smu;
    const Hist<P16> hist{smu + a.K + (size_t)per * wid};
    uint32_t* bits = hist.h + hw;
    for (int i = threadIdx.x; i < a.K + per * warps; i += blockDim.x) smu[i] = 0u;
    __syncthreads();
    for (;;) {
        const int tile = __shfl_sync(FULL, claim_warp(a.tile_counter, a.ntiles, lane), 0);
        if (tile >= a.ntiles) break;
        const int4 t = a.tiles[tile];
        wt_tile(a, t, hist, bits, nk, lane);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < a.K; k += blockDim.x) {
        const uint32_t v = nk[k];
        if (v) atomicAdd(a.n_k + k, (int)v);
    }
}

// ---------------------------------------------------------------- large-K rebuilds
// Above kLargeK topics a warp-private K-sized histogram leaves one 8-warp CTA per SM, and
// the rebuilds wait on their gathers with little else to run (halving the histogram's
// size to 16-bit counts halved both rebuilds' time).  These kernels share one histogram
// across the CTA's 256 threads and take one unit at a time (a word tile, a doc), so that
// eight CTAs per SM keep 64 warps of gathers in flight.  Their rows, counts, metadata and
// errors are those of k_wt_build / k_dt_build, bit for bit; the topic totals come from
// k_topic_totals.
constexpr int kRebuildThreads = 256;
constexpr int kSmoothMaxRounds = 2048;  // rounds of 32 topics in the smoothing table (K <= 65,536)

// Adds topics topic_of(i), i in [0, n), to the CTA's histogram (16-bit counts) and sets
// the bit of each topic whose count leaves zero; a topic >= K sets *err and is skipped.
// Four 256-token steps of loads are in flight per thread.  n is uniform across the CTA.
template <class F>
__device__ __forceinline__ void cta_hist(uint32_t n, const F& topic_of, const Hist<true>& hist, uint32_t* bits, int K,
                                         int* err) {
    for (uint32_t base = 0; base < n; base += 4u * kRebuildThreads) {
        uint32_t k[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t i = base + (uint32_t)(s * kRebuildThreads) + threadIdx.x;
            k[s] = i < n ? topic_of(i) : 0xffffffffu;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (base + (uint32_t)(s * kRebuildThreads) >= n) break;
            bool valid = k[s] != 0xffffffffu;
            uint32_t kk = k[s];
            if (valid && kk >= (uint32_t)K) {
                atomicOr(err, 1);
                valid = false;
                kk = 0xfffffffeu;
            }
            if (valid) hist_token(hist, bits, kk);
        }
    }
}

// Word-topic rows above kLargeK topics: CTA per word tile (a dense word's chunk segment
// of up to 16,384 tokens, or a sparse word over all chunks).  Shared memory: the
// histogram, the bitmap, then a sparse word's chunk segments ([C] offsets, [C + 1] prefix
// counts).  Topic totals are not accumulated here (k_topic_totals).
__global__ void __launch_bounds__(kRebuildThreads, 8) k_wt_build_cta(WtArgs a) {
    extern __shared__ uint32_t smu[];
    __shared__ uint32_t wsum[kRebuildThreads / 32];
    __shared__ int s_tile;
    const int hw = Hist<true>::words(a.K), bw = wt_bit_words(a.K);
    const Hist<true> hist{smu};
    uint32_t* bits = smu + hw;
    uint32_t* so = bits + bw;
    uint32_t* pre = so + a.C;
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < hw + bw; i += blockDim.x) smu[i] = 0u;
    for (;;) {
        __syncthreads();  // the previous tile is done with the shared state
        if (threadIdx.x == 0) {
            s_tile = (int)atomicAdd(a.tile_counter, 1u);
            last_claim_resets(a.tile_counter, s_tile, a.ntiles, (int)gridDim.x);
        }
        __syncthreads();
        const int tile = s_tile;
        if (tile >= a.ntiles) break;
        const int4 t = a.tiles[tile];
        const int w = t.x;
        if (t.w & 1) {
            const uint16_t* z = a.z + (uint32_t)t.y;
            cta_hist((uint32_t)t.z, [&](uint32_t i) { return (uint32_t)__ldg(z + i); }, hist, bits, a.K, a.err);
        } else {
            // the word's segment in every chunk, and their prefix counts
            if (threadIdx.x < 32) {
                uint32_t carry = 0;
                if (lane == 0) pre[0] = 0u;
                for (int c0 = 0; c0 < a.C; c0 += 32) {
                    const int c = c0 + lane;
                    uint32_t cnt = 0;
                    if (c < a.C) {
                        const size_t idx = (size_t)c * a.V + w;
                        so[c] = __ldg(a.seg_off + idx);
                        cnt = __ldg(a.seg_cnt + idx);
                    }
                    uint32_t incl = cnt;
#pragma unroll
                    for (int off = 1; off < 32; off <<= 1) {
                        const uint32_t v = __shfl_up_sync(FULL, incl, off);
                        if (lane >= off) incl += v;
                    }
                    if (c < a.C) pre[c + 1] = carry + incl;
                    carry += __shfl_sync(FULL, incl, 31);
                }
            }
            __syncthreads();
            const int C = a.C;
            cta_hist(pre[C], [&](uint32_t i) {
                // the chunk holding the word's i-th token: the last c with pre[c] <= i
                int lo = 0, hi = C - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (pre[mid] <= i) lo = mid; else hi = mid - 1;
                }
                return (uint32_t)__ldg(a.z + so[lo] + (i - pre[lo]));
            }, hist, bits, a.K, a.err);
        }
        __syncthreads();
        if (t.w & 1) {
            int* row = a.dwt + (size_t)w * a.K;
            cta_compact(bw, hist, bits, wsum, [&](uint32_t k, uint32_t h, uint32_t) { atomicAdd(row + k, (int)h); });
        } else {
            const int s = w - a.Vd;
            uint32_t* out = a.swt_ent + a.swt_off[s];
            const uint32_t nnz = cta_compact(bw, hist, bits, wsum,
                                             [&](uint32_t k, uint32_t h, uint32_t p) { out[p] = (k << 16) | h; });
            if (threadIdx.x == 0) a.swt_nnz[s] = nnz;
        }
    }
}

// Rows of small sparse words above kLargeK topics (at most kSmallSparse tokens, over at
// most 32 chunks): warp per word, without a histogram.  The warp holds the word's topics
// in registers (up to 8 per lane), marks them in a bitmap, gives each topic its rank among
// the word's distinct topics (the popcount prefix of the bitmap), counts per rank, and
// writes the row ascending k.  Per warp: bitmap (bw words), prefix (bw uint16) and counts
// (kSmallSparse words).  Rows equal k_wt_build_cta's.
constexpr int kSmallSparse = 256;
__host__ __device__ __forceinline__ size_t wt_small_warp_words(int K) {
    const size_t bw = (size_t)(K + 31) >> 5;
    return bw + ((bw + 1) >> 1) + kSmallSparse;
}
__global__ void __launch_bounds__(256) k_wt_sparse_small(WtArgs a) {
    extern __shared__ uint32_t smu[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bw = wt_bit_words(a.K);
    uint32_t* bits = smu + wt_small_warp_words(a.K) * wid;
    uint16_t* pre = reinterpret_cast<uint16_t*>(bits + bw);
    uint32_t* cnt = bits + bw + ((bw + 1) >> 1);
    for (int i = lane; i < bw; i += 32) bits[i] = 0u;
    for (int i = lane; i < kSmallSparse; i += 32) cnt[i] = 0u;
    __syncwarp();
    for (;;) {
        const int tile = __shfl_sync(FULL, claim_warp(a.tile_counter, a.ntiles, lane), 0);
        if (tile >= a.ntiles) break;
        const int w = a.tiles[tile].x;
        // lane c: chunk c's segment of the word, as z index minus the segment's first rank
        uint32_t so = 0, sc = 0;
        if (lane < a.C) {
            const size_t idx = (size_t)lane * a.V + w;
            so = __ldg(a.seg_off + idx);
            sc = __ldg(a.seg_cnt + idx);
        }
        uint32_t incl = sc;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, incl, off);
            if (lane >= off) incl += v;
        }
        const uint32_t base_l = so - (incl - sc);
        const uint32_t n = min(__shfl_sync(FULL, incl, 31), (uint32_t)kSmallSparse);
        uint32_t k[kSmallSparse / 32];
#pragma unroll
        for (int j = 0; j < kSmallSparse / 32; ++j) {
            const uint32_t i = 32u * (uint32_t)j + (uint32_t)lane;
            k[j] = 0xffffffffu;
            if (32u * (uint32_t)j >= n) continue;  // uniform
            // the first lane whose inclusive prefix exceeds i
            const uint32_t ii = i < n ? i : n - 1;
            int c = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t v = __shfl_sync(FULL, incl, c + step - 1);
                if (v <= ii) c += step;
            }
            const uint32_t b = __shfl_sync(FULL, base_l, c);
            if (i < n) {
                uint32_t kk = (uint32_t)__ldg(a.z + b + i);
                if (kk >= (uint32_t)a.K) {
                    atomicOr(a.err, 1);
                    kk = 0xffffffffu;
                }
                k[j] = kk;
            }
        }
#pragma unroll
        for (int j = 0; j < kSmallSparse / 32; ++j)
            if (k[j] != 0xffffffffu) atomicOr(&bits[k[j] >> 5], 1u << (k[j] & 31u));
        __syncwarp();
        uint32_t carry = 0;
        for (int wb = 0; wb < bw; wb += 32) {
            const int wi = wb + lane;
            const uint32_t c = wi < bw ? (uint32_t)__popc(bits[wi]) : 0u;
            uint32_t inc = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t v = __shfl_up_sync(FULL, inc, off);
                if (lane >= off) inc += v;
            }
            if (wi < bw) pre[wi] = (uint16_t)(carry + inc - c);
            carry += __shfl_sync(FULL, inc, 31);
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < kSmallSparse / 32; ++j) {
            const uint32_t kk = k[j];
            if (kk != 0xffffffffu) {
                const uint32_t m = bits[kk >> 5];
                atomicAdd(&cnt[pre[kk >> 5] + __popc(m & ((1u << (kk & 31u)) - 1u))], 1u);
            }
        }
        __syncwarp();
        const int s = w - a.Vd;
        uint32_t* out = a.swt_ent + a.swt_off[s];
        for (int wb = 0; wb < bw; wb += 32) {
            const int wi = wb + lane;
            uint32_t m = wi < bw ? bits[wi] : 0u;
            if (m) {
                bits[wi] = 0u;
                uint32_t p = pre[wi];
                while (m) {
                    const uint32_t kk = (uint32_t)wi * 32u + (uint32_t)(__ffs(m) - 1);
                    m &= m - 1u;
                    out[p] = (kk << 16) | cnt[p];
                    cnt[p] = 0u;
                    ++p;
                }
            }
        }
        if (lane == 0) a.swt_nnz[s] = carry;
        __syncwarp();
    }
}

// Topic totals n_k of the word tiles a.tiles (all words, or a word range): warp per tile,
// counts privatised per CTA in shared memory (K words) and flushed once; without SHARED
// (K words beyond the shared memory) the warps add to n_k directly.
template <bool SHARED>
__global__ void __launch_bounds__(256) k_topic_totals(WtArgs a) {
    extern __shared__ uint32_t smu[];
    const int lane = threadIdx.x & 31;
    if (SHARED) {
        for (int i = threadIdx.x; i < a.K; i += blockDim.x) smu[i] = 0u;
        __syncthreads();
    }
    auto add = [&](const uint16_t* z, uint32_t n) {
        for (uint32_t base = 0; base < n; base += 128) {
            uint32_t k[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const uint32_t i = base + 32u * s + lane;
                k[s] = i < n ? (uint32_t)__ldg(z + i) : 0xffffffffu;
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                if (base + 32u * s >= n) break;
                // a topic >= K is reported by the rebuild; it is not counted here
                const bool valid = k[s] < (uint32_t)a.K;
                const uint32_t kk = valid ? k[s] : 0xfffffffeu;
                if (valid && SHARED) atomicAdd(smu + kk, 1u);
                if (valid && !SHARED) atomicAdd(a.n_k + kk, 1);
            }
        }
    };
    for (;;) {
        const int tile = __shfl_sync(FULL, claim_warp(a.tile_counter, a.ntiles, lane), 0);
        if (tile >= a.ntiles) break;
        const int4 t = a.tiles[tile];
        if (t.w & 1) {
            add(a.z + (uint32_t)t.y, (uint32_t)t.z);
        } else {
            for (int c0 = 0; c0 < a.C; c0 += 32) {
                const int c = c0 + lane;
                uint32_t so = 0, sc = 0;
                if (c < a.C) {
                    const size_t idx = (size_t)c * a.V + t.x;
                    so = __ldg(a.seg_off + idx);
                    sc = __ldg(a.seg_cnt + idx);
                }
                const int nc = min(32, a.C - c0);
                for (int j = 0; j < nc; ++j) {
                    const uint32_t o = __shfl_sync(FULL, so, j), n = __shfl_sync(FULL, sc, j);
                    if (n) add(a.z + o, n);
                }
            }
        }
    }
    if (SHARED) {
        __syncthreads();
        for (int k = threadIdx.x; k < a.K; k += blockDim.x) {
            const uint32_t v = smu[k];
            if (v) atomicAdd(a.n_k + k, (int)v);
        }
    }
}

// Doc rows above kLargeK topics: CTA per doc (the doc's tokens spread over the CTA's
// threads), the histogram and bitmap shared.  Rows are ascending k with topic keys.  (Up
// to 2048 topics the warp-per-doc kernel is faster: 1.35 against 1.59 ms per sweep on the
// K=1024 corpus, where a warp's histogram is small enough for 64 warps per SM.)
__global__ void __launch_bounds__(kRebuildThreads, 8) k_dt_build_cta(DtArgs a) {
    extern __shared__ uint32_t smu[];
    __shared__ uint32_t wsum[kRebuildThreads / 32];
    const int hw = Hist<true>::words(a.K), bw = dt_bit_words(a.K);
    const Hist<true> hist{smu};
    uint32_t* bits = smu + hw;
    for (int i = threadIdx.x; i < hw + bw; i += blockDim.x) smu[i] = 0u;
    for (uint32_t d = a.d_begin + blockIdx.x; d < a.d_end; d += gridDim.x) {
        __syncthreads();  // the previous doc is done with the shared state
        const uint32_t b = __ldg(a.doc_off + d), n = __ldg(a.doc_off + d + 1) - b;
        if (n <= a.small_max) continue;  // k_dt_build_small's doc
        const uint32_t* dpos = a.dtok_pos + (b - a.tok_base);
        const uint32_t* dword = a.dtok_word + (b - a.tok_base);
        const uint16_t* z = a.z;
        cta_hist(n, [&](uint32_t i) { return (uint32_t)__ldg(z + __ldg(dpos + i)); }, hist, bits, a.K, a.err);
        __syncthreads();
        for (uint32_t base = 0; base < n; base += 4u * kRebuildThreads) {
            uint32_t pos[4], t2[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const uint32_t i = base + (uint32_t)(s * kRebuildThreads) + threadIdx.x;
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
        __syncthreads();
        uint32_t* out = a.dt_ent + (__ldg(a.dt_off + d) - a.dt_base);
        const uint32_t nnz =
            cta_compact(bw, hist, bits, wsum, [&](uint32_t k, uint32_t h, uint32_t p) { out[p] = (k << 16) | h; });
        if (threadIdx.x == 0) a.dt_nnz[d] = nnz;
    }
}

// Doc rows above kLargeK topics for docs of at most a.small_max (<= kSmallDoc) tokens:
// warp per doc, without a histogram (as k_wt_sparse_small builds small words' rows).  The
// warp holds the doc's topics in registers, marks them in a bitmap, ranks each topic among
// the doc's distinct topics by the bitmap's popcount prefix and counts per rank; a topic's
// count is then one bitmap test and one lookup, for the tokens' metadata and the row.
// Rows, metadata and errors equal k_dt_build_cta's.
constexpr int kSmallDoc = 384;
__host__ __device__ __forceinline__ size_t dt_small_warp_words(int K) {
    const size_t bw = (size_t)(K + 31) >> 5;
    return bw + ((bw + 1) >> 1) + kSmallDoc;
}
#ifndef LDA_DT_SMALL_MIN_BLOCKS
#define LDA_DT_SMALL_MIN_BLOCKS 6
#endif
__global__ void __launch_bounds__(256, LDA_DT_SMALL_MIN_BLOCKS) k_dt_build_small(DtArgs a) {
    extern __shared__ uint32_t smu[];
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bw = dt_bit_words(a.K);
    uint32_t* bits = smu + dt_small_warp_words(a.K) * wid;
    uint16_t* pre = reinterpret_cast<uint16_t*>(bits + bw);
    uint32_t* cnt = bits + bw + ((bw + 1) >> 1);
    for (int i = lane; i < bw; i += 32) bits[i] = 0u;
    for (int i = lane; i < kSmallDoc; i += 32) cnt[i] = 0u;
    __syncwarp();
    // the doc's count of topic k (bits, pre and cnt complete)
    auto count_of = [&](uint32_t k) -> uint32_t {
        if (k >= (uint32_t)a.K) return 0u;
        const uint32_t m = bits[k >> 5], sh = k & 31u;
        return (m >> sh) & 1u ? cnt[pre[k >> 5] + __popc(m & ((1u << sh) - 1u))] : 0u;
    };
    for (uint32_t d = a.d_begin + blockIdx.x * warps + wid; d < a.d_end; d += gridDim.x * warps) {
        const uint32_t b = __ldg(a.doc_off + d), n = __ldg(a.doc_off + d + 1) - b;
        if (n > a.small_max) continue;  // k_dt_build_cta's doc
        const uint32_t* dpos = a.dtok_pos + (b - a.tok_base);
        const uint32_t* dword = a.dtok_word + (b - a.tok_base);
        uint32_t k[kSmallDoc / 32];
#pragma unroll
        for (int j = 0; j < kSmallDoc / 32; ++j) {
            const uint32_t i = 32u * (uint32_t)j + (uint32_t)lane;
            k[j] = i < n ? __ldg(dpos + i) : 0xffffffffu;
        }
#pragma unroll
        for (int j = 0; j < kSmallDoc / 32; ++j) {
            if (k[j] == 0xffffffffu) continue;
            uint32_t kk = (uint32_t)__ldg(a.z + k[j]);
            if (kk >= (uint32_t)a.K) {
                atomicOr(a.err, 1);
                kk = 0xffffffffu;
            }
            k[j] = kk;
        }
#pragma unroll
        for (int j = 0; j < kSmallDoc / 32; ++j)
            if (k[j] != 0xffffffffu) atomicOr(&bits[k[j] >> 5], 1u << (k[j] & 31u));
        __syncwarp();
        uint32_t carry = 0;
        for (int wb = 0; wb < bw; wb += 32) {
            const int wi = wb + lane;
            const uint32_t c = wi < bw ? (uint32_t)__popc(bits[wi]) : 0u;
            uint32_t inc = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t v = __shfl_up_sync(FULL, inc, off);
                if (lane >= off) inc += v;
            }
            if (wi < bw) pre[wi] = (uint16_t)(carry + inc - c);
            carry += __shfl_sync(FULL, inc, 31);
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < kSmallDoc / 32; ++j) {
            const uint32_t kk = k[j];
            if (kk != 0xffffffffu) {
                const uint32_t m = bits[kk >> 5];
                atomicAdd(&cnt[pre[kk >> 5] + __popc(m & ((1u << (kk & 31u)) - 1u))], 1u);
            }
        }
        __syncwarp();
        // each token's counts of its word's max and 2nd topics
        for (uint32_t base = 0; base < n; base += 32) {
            const uint32_t i = base + (uint32_t)lane;
            if (i < n) {
                const uint32_t pos = __ldg(dpos + i), t2 = __ldg(a.st_top2 + __ldg(dword + i));
                a.meta[pos - a.tok_base] = (count_of(t2 >> 16) << 16) | count_of(t2 & 0xffffu);
            }
        }
        __syncwarp();
        uint32_t* out = a.dt_ent + (__ldg(a.dt_off + d) - a.dt_base);
        for (int wb = 0; wb < bw; wb += 32) {
            const int wi = wb + lane;
            uint32_t m = wi < bw ? bits[wi] : 0u;
            if (m) {
                bits[wi] = 0u;
                uint32_t p = pre[wi];
                while (m) {
                    const uint32_t kk = (uint32_t)wi * 32u + (uint32_t)(__ffs(m) - 1);
                    m &= m - 1u;
                    out[p] = (kk << 16) | cnt[p];
                    cnt[p] = 0u;
                    ++p;
                }
            }
        }
        if (lane == 0) a.dt_nnz[d] = carry;
        __syncwarp();
    }
}

// The sweep's reciprocals, base column and topic order (recip_order): CTA per 32 topics, K
// floats of shared memory.
__global__ void __launch_bounds__(kRecipThreads) k_recip_order(const int* __restrict__ n_k, int K, float Vbeta,
                                                               float beta, float* recip, float* base, int* order) {
    extern __shared__ float smf[];
    recip_order(n_k, K, Vbeta, beta, recip, base, order, (int)blockIdx.x * 32, smf);
}

// Word statistics: warp per word.
__global__ void __launch_bounds__(256) k_word_stats(StatsArgs a) {
    extern __shared__ float smf[];
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* col = smf + (size_t)stats_warp_words(a.K) * wid;
    uint32_t* bits = reinterpret_cast<uint32_t*>(col + ((a.K + 3) & ~3));
    bool clean = false;
    NoTokenStats none;
    for (int w = a.wlo + blockIdx.x * warps + wid; w < a.V; w += gridDim.x * warps)
        word_stats_word(a, w, col, bits, clean, none, lane);
}

// Word statistics of dense words above kLargeK topics: CTA per word, with the word's column
// in shared memory (K floats), formed by all threads.  The top three are merged over the
// warps; the serial Q sums are warp 0's while the other warps take the rounds of the Q-round
// table.  (A warp per word read its count row three times, 313 dependent steps each at
// K=10,000: 141 us for 1,200 words, with one such CTA of 8 words per SM.)
//
// The Q-round table of word w (a.qtab): for lane slot ls and round r, the Kogge-Stone total
// and largest prefix of alpha * colz(ls + 32 * (32 r + l)), l = 0..31 (slots past the lane
// slot's last topic add 0, colz the column with its max topic zeroed), then per lane slot the
// carries as the fadd chain of the totals: entry (ls, r) = (carry before round r, carry + the
// round's largest prefix).  Lane ls scans its own slot's 32 terms of a round serially in
// Kogge-Stone order.
__global__ void __launch_bounds__(256) k_word_stats_dense_cta(StatsArgs a) {
    extern __shared__ float smf[];
    __shared__ float sv[24];
    __shared__ int sk[24];
    __shared__ float2 tot[16 * 32];  // qtab_rounds(K) <= 16
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, K = a.K;
    float* col = smf;
    for (int w = a.wlo + blockIdx.x; w < a.V; w += gridDim.x) {
        const int* row = a.dwt + (size_t)w * K;
        float a1 = -1.0f, a2 = -1.0f, a3 = -1.0f;
        int i1 = 0x7fffffff, i2 = 0x7fffffff, i3 = 0x7fffffff;
        for (int b = threadIdx.x; b < K; b += 4 * 256) {
            int c[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) c[j] = b + 256 * j < K ? __ldg(row + b + 256 * j) : 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = b + 256 * j;
                if (k >= K) break;
                const float x = fmul(fadd(__int2float_rn(c[j]), a.beta), __ldg(a.recip + k));
                col[k] = x;
                top3_insert(x, k, a1, i1, a2, i2, a3, i3);
            }
        }
        float v[3];
        int kk[3];
        warp_top3(a1, i1, a2, i2, a3, i3, v, kk);
        if (lane < 3) {
            sv[3 * wid + lane] = lane == 0 ? v[0] : lane == 1 ? v[1] : v[2];
            sk[3 * wid + lane] = lane == 0 ? kk[0] : lane == 1 ? kk[1] : kk[2];
        }
        __syncthreads();
        if (wid == 0) {
            warp_top3(lane < 24 ? sv[lane] : -1.0f, lane < 24 ? sk[lane] : 0x7fffffff, -1.0f, 0x7fffffff, -1.0f,
                      0x7fffffff, v, kk);
            if (lane == 0) col[kk[0]] = 0.0f;  // fmaf(alpha, 0, q) is q: the max topic adds nothing
        }
        __syncthreads();
        if (wid == 0) {
            float ql = 0.0f;
#pragma unroll 8
            for (int k = lane; k < K; k += 32) ql = ffma(a.alpha, col[k], ql);
            const float Q = __shfl_sync(FULL, warp_ks_scan(ql, lane), 31);
            a.st_ql[(size_t)w * 32 + lane] = ql;
            if (lane == 0) {
                a.st_top2[w] = ((uint32_t)kk[1] << 16) | (uint32_t)kk[0];
                a.st_k3[w] = (uint32_t)kk[2];
                a.st_phi[w] = make_float4(v[0], v[1], v[2], Q);
            }
        } else if (a.qtab) {
            const uint32_t n = (uint32_t)((K - lane + 31) / 32);
            for (int r = wid - 1; r < a.qrounds; r += 7) {
                float t[32];
#pragma unroll
                for (int l = 0; l < 32; ++l) {
                    const uint32_t i = 32u * (uint32_t)r + (uint32_t)l;
                    t[l] = i < n ? fmul(a.alpha, col[lane + 32 * (int)i]) : 0.0f;
                }
                thread_ks_scan(t);
                float mx = t[0];
#pragma unroll
                for (int l = 1; l < 32; ++l) mx = fmaxf(mx, t[l]);
                tot[32 * r + lane] = make_float2(t[31], mx);
            }
        }
        __syncthreads();
        if (wid == 1 && a.qtab) {
            float2* tab = a.qtab + ((size_t)w * 32 + lane) * a.qrounds;
            float carry = 0.0f;
            for (int r = 0; r < a.qrounds; ++r) {
                const float2 x = tot[32 * r + lane];
                tab[r] = make_float2(carry, fadd(carry, x.y));
                carry = fadd(carry, x.x);
            }
        }
    }
}

// Doc-topic rebuild: warp per doc of one chunk.  P16: 16-bit histogram counts (a doc has
// at most 65,535 tokens).
template <bool P16>
__global__ void __launch_bounds__(256) k_dt_build(DtArgs a) {
    extern __shared__ uint32_t smu[];
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hw = Hist<P16>::words(a.K);
    const int per = hw + dt_bit_words(a.K);
    const Hist<P16> hist{smu + (size_t)per * wid};
    uint32_t* bits = hist.h + hw;
    for (int i = threadIdx.x; i < per * warps; i += blockDim.x) smu[i] = 0u;
    __syncthreads();
    for (uint32_t d = a.d_begin + blockIdx.x * warps + wid; d < a.d_end; d += gridDim.x * warps) {
        dt_doc(a, d, hist, bits, lane);
    }
}

// Sampler: warp per tile, tiles taken from an atomic counter (the next one is claimed when a
// tile starts, so that the claim's round trip overlaps the tile's work).  SKEWKEYS: the doc
// rows' keys are byte offsets of word-column slots and a.base is there (the trainer's rows
// and tables up to kLargeK topics).
template <bool LL, int QB = 1, bool SKEWKEYS = true>
__global__ void __launch_bounds__(32 * kSampleWarps, QB > 1 ? LDA_SAMPLE_QB_MIN_BLOCKS
                                                       : (!LL ? LDA_SAMPLE_MIN_BLOCKS : QB == 0 ? kSampleLL0MinBlocks : LDA_SAMPLE_LL_MIN_BLOCKS))
k_sample_t(SampleArgs a) {
    extern __shared__ float smf[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* col = smf + (size_t)sample_warp_words(a.K, a.nslots) * wid;
    float* slots = col + col_words(a.K);
    uint32_t* ctr = reinterpret_cast<uint32_t*>(slots + ((row_state_words(a.nslots) + 3) & ~3));
    if (lane < C_NUM) ctr[lane] = 0u;
    __syncwarp();
    int held = kHoldsNone;
    int tile = __shfl_sync(FULL, claim_warp(a.tile_counter, a.ntiles, lane), 0);
    while (tile < a.ntiles) {
        const int next = claim_warp(a.tile_counter, a.ntiles, lane);
        sample_tile<LL, QB, SKEWKEYS>(a, tile, a.tiles[tile], a.iter, col, slots, held, ctr, lane);
        tile = __shfl_sync(FULL, next, 0);
    }
    __syncwarp();
    if (lane < C_NUM && ctr[lane]) atomicAdd(a.ctr + lane, (unsigned long long)ctr[lane]);
}

// ------------------------------------------------------------------ large K
// Above kLargeK topics a per-warp word column (4K bytes) leaves few warps on an SM, so
// the sampler splits a chunk's tiles by kind.  Dense words: one CTA per tile, its warps
// share one column in shared memory and take the tile's 32-token groups in turn.  Sparse
// words: warp per tile with no column at all (ColBits).  Both run the same per-group code
// (sample_groups) on the same values as the per-warp column, so results are unchanged.
// The threshold is kLargeK (sweep_body.cuh).

// Sparse-word view without a column: beta * r_k for every topic in shared memory (the CTA's),
// the word's topics as a bitmap with the number of them before each 32-topic word; a topic's
// count is read from the word's row (ascending k), and phi_k is formed exactly as a column
// forms it.  The max topic's bit is set too, so that one test finds every topic whose value
// is not beta * r_k.
struct ColBits {
    using Entry = uint32_t;  // a doc-row entry: (k << 16) | count
    static constexpr bool kAhead = false, kOwnMass = true;
    const uint32_t* bits;  // ceil(K/32) words
    const uint16_t* pre;   // the word's topics before each of them
    const uint32_t* ent;   // the word's row, (k << 16) | count
    const float* base;     // beta * r_k in the skewed layout: at col_skew(k)
    const float* __restrict__ recip;
    float beta;
    int maxK;
    bool extra;            // the max topic is not one of the word's
    bool rich;             // the word holds more than a 32nd of the topics
    // the place in the word's row of a topic with its bit set (not the max topic unless it is
    // one of the word's)
    __device__ __forceinline__ uint32_t place(int k, uint32_t b) const {
        uint32_t i = pre[k >> 5] + __popc(b & ((1u << (k & 31)) - 1u));
        if (extra && (maxK >> 5) == (k >> 5) && maxK < k) --i;
        return i;
    }
    // phi_k of a topic with its bit set
    __device__ __forceinline__ float marked(int k, uint32_t b) const {
        if (k == maxK) return 0.0f;
        return fmul(fadd(u2f(__ldg(ent + place(k, b)) & 0xffffu), beta), __ldg(recip + k));
    }
    __device__ __forceinline__ float operator()(int k) const {
        const uint32_t b = bits[k >> 5];
        return (b >> (k & 31)) & 1u ? marked(k, b) : base[col_skew(k)];
    }
    __device__ __forceinline__ float row(uint32_t key) const { return (*this)((int)key); }
    __device__ __forceinline__ int topic(uint32_t key) const { return (int)key; }
    __device__ __forceinline__ uint32_t key(uint32_t e) const { return e >> 16; }
    __device__ __forceinline__ float cnt(uint32_t e) const { return u2f(e & 0xffffu); }
    // A lane's sum over a row's entries l, l + 32, ... (lane_mass): four steps' lookups first,
    // then the marked topics' values, so that no branch keeps the lookups apart: one by one
    // when they are seldom (most sparse words hold a few of the thousands of topics), and
    // four at a time with their loads together when the word is rich in topics (3.5M tokens
    // of 7,000 words at K=3000, early: one by one made a sweep a quarter slower than a
    // predicated lookup per entry).  One body for full and partial
    // batches: with the straight-line tails of the column samplers and a lookup of marked
    // topics in each, the kernel missed the instruction cache.
    __device__ __forceinline__ float mass(const uint32_t* __restrict__ row, uint32_t lane, uint32_t nnz) const {
        float acc = 0.0f;
        for (uint32_t q = lane; q < nnz + lane; q += 128u) {
            uint32_t e[4], hit = 0u, bw[4];
            float ph[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) e[j] = q + 32u * j < nnz ? __ldg(row + q + 32u * j) : 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = (int)key(e[j]);
                bw[j] = bits[k >> 5];
                ph[j] = base[col_skew(k)];
                hit |= ((bw[j] >> (k & 31)) & 1u) << j;
            }
            if (rich && hit) {
                uint32_t en[4];
                float rk[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int k = (int)key(e[j]);
                    const bool in = (hit >> j) & 1u && k != maxK;
                    en[j] = in ? __ldg(ent + place(k, bw[j])) : 0u;
                    rk[j] = in ? __ldg(recip + k) : 0.0f;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if ((hit >> j) & 1u)
                        ph[j] = (int)key(e[j]) == maxK ? 0.0f : fmul(fadd(u2f(en[j] & 0xffffu), beta), rk[j]);
                hit = 0u;
            }
            while (hit) {
                const int j = __ffs(hit) - 1;
                hit &= hit - 1u;
                const uint32_t ej = j == 0 ? e[0] : j == 1 ? e[1] : j == 2 ? e[2] : e[3];
                const uint32_t bj = j == 0 ? bw[0] : j == 1 ? bw[1] : j == 2 ? bw[2] : bw[3];
                const float v = marked((int)key(ej), bj);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i == j) ph[i] = v;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) acc = ffma(cnt(e[j]), ph[j], acc);
        }
        return acc;
    }
};

__host__ __device__ __forceinline__ int large_bit_words(int K) { return (K + 31) >> 5; }
__host__ __device__ __forceinline__ int large_pre_words(int K) { return ((K + 31) >> 5) + 1 & ~1; }

// Shared memory of the sparse-word kernel: beta * r_k in the skewed column layout
// (col_words(K) floats) and the smoothing table's round ends, then per warp the bitmap, the
// prefix counts (uint16, an even number), the counter row, the row state and the 32 prefixes
// of a one-round word's own Q terms.
__host__ __device__ __forceinline__ int smooth_rounds(int K) { return (K + 31) >> 5; }
__host__ __device__ __forceinline__ int sparse_large_warp_words(int K, int nslots) {
    return ((large_bit_words(K) + large_pre_words(K) / 2 + C_NUM + 32 + 1) & ~1) + row_state_words(nslots);
}
__host__ __device__ __forceinline__ size_t sparse_large_smem(int K, int warps, int nslots) {
    return (size_t)(col_words(K) + ((smooth_rounds(K) + 1) & ~1) + warps * sparse_large_warp_words(K, nslots)) * 4;
}

// Shared memory of the dense-word sampler: the word column, the warps' counter rows, their
// LL partials and (when qtab_rounds(K) > 0) the Q-round table of 32 x R float2.
__host__ __device__ __forceinline__ size_t dense_large_smem(int K, int warps, int nslots) {
    return (((size_t)col_words(K) * 4 + (size_t)warps * C_NUM * 4 + 7) & ~(size_t)7) + (size_t)warps * 8 +
           (size_t)32 * qtab_rounds(K) * sizeof(float2) + (size_t)warps * row_state_words(nslots) * 4;
}

// Warps per CTA of the two samplers and the CTAs per SM they are compiled for.  Dense: the
// CTAs share the SM's registers four ways (64 a thread) so that one CTA's column build and
// tile end overlap the others' sampling; fewer, larger CTAs with more row slots lose (10M
// tokens at K=10,000: 4.79 ms per sweep against 5.05 with two CTAs of 16 warps, 5.07 with
// three of 8).  Sparse: the reciprocals (41 KB at K=10,000) are the CTA's, so two CTAs of 12
// warps hold as many warps as three of 8, and 80 registers a thread avoid 130 bytes of
// spills (5.40 -> 4.79 ms with the dense kernel as it is; 16 warps at 64 registers 5.6).
#ifndef LDA_DENSE_LARGE_MIN_BLOCKS
#define LDA_DENSE_LARGE_MIN_BLOCKS 4
#endif
#ifndef LDA_SPARSE_LARGE_MIN_BLOCKS
#define LDA_SPARSE_LARGE_MIN_BLOCKS 2
#endif
constexpr int kDenseWarps = 8, kSparseWarps = 12;

// The sparse-word sampler keeps each word's Qw rounds' table in registers (lane r: round
// r), so a Q draw evaluates the one round that holds its target instead of walking them.
template <bool LL, int QB>
__global__ void __launch_bounds__(32 * kSparseWarps, LDA_SPARSE_LARGE_MIN_BLOCKS) k_sample_sparse_large(SampleArgs a) {
    extern __shared__ float smf[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bw = large_bit_words(a.K), pw = large_pre_words(a.K);
    float* base = smf;
    float* tend = smf + col_words(a.K);
    const int rounds = smooth_rounds(a.K);
    uint32_t* bits = reinterpret_cast<uint32_t*>(tend + ((rounds + 1) & ~1)) + (size_t)sparse_large_warp_words(a.K, a.nslots) * wid;
    float* slots = reinterpret_cast<float*>(bits);
    bits += row_state_words(a.nslots);
    uint16_t* pre = reinterpret_cast<uint16_t*>(bits + bw);
    uint32_t* ctr = bits + bw + pw / 2;
    float* wp = reinterpret_cast<float*>(ctr + C_NUM);
    for (int k = threadIdx.x; k < a.K; k += blockDim.x) base[col_skew(k)] = fmul(a.beta, __ldg(a.recip + k));
    for (int i = threadIdx.x; i < rounds; i += blockDim.x) tend[i] = __ldg(a.smooth + min(a.K, 32 * i + 32) - 1);
    for (int i = lane; i < bw; i += 32) bits[i] = 0u;
    if (lane < C_NUM) ctr[lane] = 0u;
    __syncthreads();
    // the next tile is claimed when a tile starts, so that the claim's round trip overlaps
    // the tile's work
    int tile = __shfl_sync(FULL, claim_warp(a.tile_counter, a.ntiles, lane), 0);
    for (;;) {
        if (tile >= a.ntiles) break;
        const int next = claim_warp(a.tile_counter, a.ntiles, lane);
        const int4 t = a.tiles[tile];
        const int w = t.x;
        const int s = w - a.Vd;
        const uint32_t* ent = a.swt_ent + __ldg(a.swt_off + s);
        const uint32_t nnz_w = __ldg(a.swt_nnz + s);
        // the word's statistics, loaded before the bitmap work so that their loads overlap it
        const int maxK = (int)(__ldg(a.st_top2 + w) & 0xffffu);
        const float4 ph = __ldg(a.st_phi + w);
        const float QL = __ldg(a.st_ql + (size_t)w * 32 + lane);
        // the word's topics into the bitmap; pre[j] = the rank of the first of the word's
        // topics in bitmap word j (the entries ascend, so that is the entry's index).  Only
        // words with a set bit are ever read, so the others are left as they are.
        for (uint32_t e = lane; e < nnz_w; e += 32) {
            const uint32_t k = __ldg(ent + e) >> 16;
            atomicOr(&bits[k >> 5], 1u << (k & 31u));
            if (e == 0 || (__ldg(ent + e - 1) >> 21) != (k >> 5)) pre[k >> 5] = (uint16_t)e;
        }
        __syncwarp();
        const bool extra = !((bits[maxK >> 5] >> (maxK & 31)) & 1u);
        __syncwarp();
        if (lane == 0) {
            if (extra) bits[maxK >> 5] |= 1u << (maxK & 31);
            ctr[C_WNNZ] += nnz_w;
            ctr[C_TSPARSE] += 1u;
        }
        const float QP = warp_ks_scan(QL, lane);
        const float Q = __shfl_sync(FULL, QP, 31);
        __syncwarp();
        const ColBits view{bits, pre, ent, base, a.recip, a.beta, maxK, extra, nnz_w > (uint32_t)a.K >> 5};
        SplitQ sq{ent, nnz_w, __shfl_sync(FULL, QL, 0), a.smooth, a.recip};
        if (nnz_w <= 32u) {
            // the one round's prefixes, for thread_split_draw
            int key;
            float term = 0.0f;
            bool ok = false;
            if ((uint32_t)lane < nnz_w) sq.slot((uint32_t)lane, maxK, a.alpha, key, term, ok);
            wp[lane] = warp_ks_scan(term, lane);
            sq.wp = wp;
            sq.wok = __ballot_sync(FULL, ok);
        }
        sq.tend = tend;
        split_q_table(sq, maxK, a.alpha, lane);
        double ll = sample_groups<LL, QB, true>(a, (uint32_t)t.y, (uint32_t)t.z, 0u, 32u, a.iter,
                                                                    maxK, ph, QL, QP, Q, view, ctr, lane, slots,
                                                                    nullptr, 0, &sq);
        if (LL) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) ll += __shfl_xor_sync(FULL, ll, off);
            if (lane == 0) a.tile_ll[tile] = ll;
        }
        __syncwarp();
        for (uint32_t e = lane; e < nnz_w; e += 32) bits[(__ldg(ent + e) >> 16) >> 5] = 0u;
        if (lane == 0) bits[maxK >> 5] = 0u;
        __syncwarp();
        tile = __shfl_sync(FULL, next, 0);
    }
    __syncwarp();
    if (lane < C_NUM && ctr[lane]) atomicAdd(a.ctr + lane, (unsigned long long)ctr[lane]);
}

template <bool LL, int QB>
__global__ void __launch_bounds__(32 * kDenseWarps, LDA_DENSE_LARGE_MIN_BLOCKS) k_sample_dense_large(SampleArgs a) {
    extern __shared__ float smf[];
    __shared__ int s_tile;
    __shared__ uint32_t s_group;  // plain sweeps: the tile's next 32-token group
    __shared__ float s_qps[32];   // the word's Q prefixes
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* col = smf;
    uint32_t* ctr_all = reinterpret_cast<uint32_t*>(col + col_words(a.K));
    uint32_t* ctr = ctr_all + C_NUM * wid;
    double* wll = reinterpret_cast<double*>(
        (reinterpret_cast<uintptr_t>(ctr_all + C_NUM * warps) + 7) & ~(uintptr_t)7);
    const int qr = qtab_rounds(a.K);
    float2* qtab = reinterpret_cast<float2*>(wll + warps);
    float* slots = reinterpret_cast<float*>(qtab + 32 * qr) + (size_t)row_state_words(a.nslots) * wid;
    if (lane < C_NUM) ctr[lane] = 0u;
    __syncthreads();
    for (;;) {
        if (threadIdx.x == 0) {
            s_tile = (int)atomicAdd(a.tile_counter, 1u);
            last_claim_resets(a.tile_counter, s_tile, a.ntiles, (int)gridDim.x);
        }
        __syncthreads();
        const int tile = s_tile;
        if (tile >= a.ntiles) break;
        const int4 t = a.tiles[tile];
        const int w = t.x;
        const int* wrow = a.dwt + (size_t)w * a.K;
        // phi_k = ((float)n_wk + beta) * r_k with r_k = 1 / ((float)n_k + V*beta), the values
        // of the per-warp columns
        // the count row is read once per tile and chunk (800 MB per chunk on the K=10,000
        // corpus): evict_first, so that it displaces fewer of the chunk's doc rows in L2
        // (that corpus: samplers 116.1 -> 115.6 ms per sweep)
        const uint64_t spol = l2_stream_policy();
        for (int k = threadIdx.x; k < a.K; k += blockDim.x) {
            const float rk = __ldg(a.recip + k);
            const int c = ldg_hint(wrow + k, spol);
            col[col_skew(k)] = fmul(fadd(__int2float_rn(c), a.beta), rk);
        }
        const int maxK = (int)(__ldg(a.st_top2 + w) & 0xffffu);
        __syncthreads();
        if (threadIdx.x == 0) {
            col[col_skew(maxK)] = 0.0f;
            ctr[C_TDENSE] += 1u;
            s_group = 0u;
        }
        __syncthreads();
        if (qr) {
            // the word's Q-round table, built by the word statistics
            const float2* src = a.qtab_g + (size_t)w * 32 * qr;
            for (int i = threadIdx.x; i < 32 * qr; i += blockDim.x) qtab[i] = __ldg(src + i);
            __syncthreads();
        }
        const float4 ph = __ldg(a.st_phi + w);
        const float QL = __ldg(a.st_ql + (size_t)w * 32 + lane);
        const float QP = warp_ks_scan(QL, lane);
        const float Q = __shfl_sync(FULL, QP, 31);
        if (threadIdx.x < 32) s_qps[lane] = QP;
        __syncthreads();
        double ll = sample_groups<LL, QB, false>(a, (uint32_t)t.y, (uint32_t)t.z, 32u * wid,
                                                                     32u * warps, a.iter, maxK, ph, QL, QP, Q,
                                                                     ColShared{col}, ctr, lane, slots,
                                                                     qr ? qtab : nullptr, qr, nullptr,
                                                                     LL ? nullptr : &s_group, s_qps);
        if (LL) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) ll += __shfl_xor_sync(FULL, ll, off);
            if (lane == 0) wll[wid] = ll;
        }
        __syncthreads();
        if (LL && threadIdx.x == 0) {
            double sum = 0.0;
            for (int i = 0; i < warps; ++i) sum += wll[i];
            a.tile_ll[tile] = sum;
        }
    }
    __syncwarp();
    if (lane < C_NUM && ctr[lane]) atomicAdd(a.ctr + lane, (unsigned long long)ctr[lane]);
}

// ------------------------------------------------------------ large-K word statistics
// For K > kLargeK a sparse word's column is beta * r_k except at its own few topics, so its
// statistics need no column: the top three come from its own topics and the first three
// other topics of the CTA's list of topics in decreasing beta * r_k (ties to the lower k),
// and its split Q from its own entries and the smoothing table (Qw in st_ql slot 0, Qs in
// slot 1).  Dense words take k_word_stats_dense_cta.
// Shared memory of the sparse-word statistics: the order list, then per warp the bitmap.
// The reciprocals are read from the global table (k_recip_order), so that the CTA does not
// hold K of them and eight CTAs fit per SM.
__host__ __device__ __forceinline__ size_t stats_sparse_smem(int K, int warps) {
    return kOrderList * 4 + (size_t)warps * (large_bit_words(K) * 4);
}

__global__ void __launch_bounds__(256) k_word_stats_sparse_large(StatsArgs a) {
    extern __shared__ float smf[];
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bw = large_bit_words(a.K);
    const float* __restrict__ r = a.recip;
    int* order = reinterpret_cast<int*>(smf);
    uint32_t* bits = reinterpret_cast<uint32_t*>(order + kOrderList) + (size_t)bw * wid;
    const int L = min(kOrderList, a.K);
    for (int i = threadIdx.x; i < L; i += blockDim.x) order[i] = __ldg(a.order + i);
    for (int i = lane; i < bw; i += 32) bits[i] = 0u;
    __syncthreads();
    for (int w = max(a.Vd, a.wlo) + blockIdx.x * warps + wid; w < a.V; w += gridDim.x * warps) {
        const int s = w - a.Vd;
        const uint32_t* ent = a.swt_ent + __ldg(a.swt_off + s);
        const uint32_t nnz = __ldg(a.swt_nnz + s);
        float a1 = -1.0f, a2 = -1.0f, a3 = -1.0f;
        int i1 = 0x7fffffff, i2 = 0x7fffffff, i3 = 0x7fffffff;
        for (uint32_t e = lane; e < nnz; e += 32) {
            const uint32_t en = __ldg(ent + e);
            const int k = (int)(en >> 16);
            atomicOr(&bits[k >> 5], 1u << (k & 31));
            top3_insert(fmul(fadd(u2f(en & 0xffffu), a.beta), r[k]), k, a1, i1, a2, i2, a3, i3);
        }
        __syncwarp();
        // with the best three topics outside the word
        top3_outside(a, order, bits, a1, i1, a2, i2, a3, i3, lane);
        float v[3];
        int kk[3];
        warp_top3(a1, i1, a2, i2, a3, i3, v, kk);
        const int k1 = kk[0];
        // Q = Qw + Qs (the split Q bucket): Qw over the word's own topics in rounds of 32
        // entries (ascending k, the max topic's term 0), Qs = T[K-1] - sm_max
        float carry = 0.0f;
        for (uint32_t base = 0; base < nnz; base += 32) {
            const uint32_t e = base + (uint32_t)lane;
            float term = 0.0f;
            if (e < nnz) {
                const uint32_t en = __ldg(ent + e);
                const int k = (int)(en >> 16);
                if (k != k1) term = fmul(a.alpha, fmul(u2f(en & 0xffffu), r[k]));
            }
            const float P = fadd(carry, warp_ks_scan(term, lane));
            carry = __shfl_sync(FULL, P, 31);
        }
        const float Qw = carry;
        const float Qs = fsub(__ldg(a.smooth + a.K - 1), fmul(a.alpha, fmul(a.beta, r[k1])));
        a.st_ql[(size_t)w * 32 + lane] = lane == 0 ? Qw : (lane == 1 ? Qs : 0.0f);
        if (lane == 0) {
            a.st_top2[w] = ((uint32_t)kk[1] << 16) | (uint32_t)k1;
            a.st_k3[w] = (uint32_t)kk[2];
            a.st_phi[w] = make_float4(v[0], v[1], v[2], fadd(Qw, Qs));
        }
        __syncwarp();
        for (uint32_t e = lane; e < nnz; e += 32) bits[(__ldg(ent + e) >> 16) >> 5] = 0u;
        __syncwarp();
    }
}

// The smoothing table of the split Q bucket (K > kLargeK): T[k] = carry + Kogge-Stone scan
// of sm_k = alpha * (beta * r_k) over rounds of 32 topics, the carry being the previous
// round's last prefix, so T ascends but for rounding and T[K-1] is the total.  r_k is formed from
// n_k as k_recip_order forms it.  One CTA: its warps scan the rounds in parallel (the scan of
// a round does not depend on the carry), one thread chains the carries, then every T[k] is
// one addition.  T holds each round's scan until the carries are known.
__global__ void __launch_bounds__(1024) k_smooth_table(const int* __restrict__ n_k, int K, float Vbeta, float alpha,
                                                       float beta, float* __restrict__ T) {
    __shared__ float carry_s[kSmoothMaxRounds];
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rounds = (K + 31) >> 5;
    for (int rd = wid; rd < rounds; rd += warps) {
        const int k = 32 * rd + lane;
        const float sm = k < K ? fmul(alpha, fmul(beta, __fdiv_rn(1.0f, fadd(__int2float_rn(n_k[k]), Vbeta)))) : 0.0f;
        const float sc = warp_ks_scan(sm, lane);
        if (k < K) T[k] = sc;
        if (lane == 31) carry_s[rd] = sc;  // the round's total for now
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float carry = 0.0f;
        for (int rd = 0; rd < rounds; ++rd) {
            const float tot = carry_s[rd];
            carry_s[rd] = carry;
            carry = fadd(carry, tot);
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += blockDim.x) T[k] = fadd(carry_s[k >> 5], T[k]);
}

// Fixed-order FP64 reduction of the per-tile LL partials (one CTA of 1024 threads).
// Replaces LDATrainPerplexityReduce (EZLDA/utility.cu:2106-2151).
__global__ void __launch_bounds__(1024) k_ll_reduce(const double* __restrict__ in, int n, double* out) {
    __shared__ double s[1024];
    const double acc = strided_sum(in, n);
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int h = blockDim.x >> 1; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = s[0];
}

}  // namespace dev
}  // namespace lda
