// serving.cu -- fold-in of new documents against a frozen model, with continuous batching.
//
// EZLDA has no inference path.  Fold-in is its sweep with the word-topic side frozen: the
// conditional of a token of word w in a new document d is p(k) ∝ (n_dk+alpha)*phi_wk, with
// phi_wk = (n_wk+beta)/(n_k+V*beta) from the trained counts and n_dk the document's own
// counts at the start of each sweep.  The draw uses the same decomposition and arithmetic
// as the training sampler (max topic / S over the document's row / Q bucket, early accept).
//
// Device layout of a server: a token pool (word + topic per token, each request a
// contiguous range), a row pool (up to K entries per request slot: the request's topic counts
// at the start of the sweep) and a request table.  A step runs one sweep for every active request (each at its own sweep
// index); requests that arrive while others run are admitted at the next step when the
// token pool and the slots have room.  Each request's randoms are keyed on (seed, request
// id, sweep, position), so its result does not depend on what it was batched with.
#include <algorithm>
#include <chrono>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <thread>
#include <vector>

#include "common.h"
#include "launch_util.h"
#include "sweep_body.cuh"

using namespace lda;

namespace lda {
namespace dev {

// Dense phi of every word, phi_wk = ((float)n_wk + beta) * r_k, r_k = 1/((float)n_k + V*beta)
// (the same column the sweep builds per tile).
struct PhiArgs {
    int V, Vd, K;
    float beta, Vbeta;
    const int* n_k;
    const int* dwt;
    const uint32_t* swt_off;
    const uint32_t* swt_nnz;
    const uint32_t* swt_ent;
    float* phi;
};

__global__ void __launch_bounds__(256) k_phi_dense(PhiArgs a) {
    extern __shared__ float smf[];
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* r = smf;
    fill_recip(r, a.n_k, a.K, a.Vbeta);
    __syncthreads();
    for (int w = blockIdx.x * warps + wid; w < a.V; w += gridDim.x * warps) {
        float* out = a.phi + (size_t)w * a.K;
        if (w < a.Vd) {
            const int* row = a.dwt + (size_t)w * a.K;
            for (int k = lane; k < a.K; k += 32) out[k] = fmul(fadd(__int2float_rn(__ldg(row + k)), a.beta), r[k]);
        } else {
            for (int k = lane; k < a.K; k += 32) out[k] = fmul(a.beta, r[k]);
            __syncwarp();
            const int s = w - a.Vd;
            const uint32_t off = __ldg(a.swt_off + s), nnz = __ldg(a.swt_nnz + s);
            for (uint32_t e = lane; e < nnz; e += 32) {
                const uint32_t en = __ldg(a.swt_ent + off + e);
                out[en >> 16] = fmul(fadd(u2f(en & 0xffffu), a.beta), r[en >> 16]);
            }
        }
        __syncwarp();
    }
}

// Above kLargeK topics the trainer's statistics give a sparse word its split Q bucket
// ({Qw, Qs} in the lane-partial slots); the frozen model has no sparse word rows, so its
// sparse words get the lane partials back, formed from the dense phi rows as k_word_stats
// forms them from a column (serial fmaf of alpha * phi_k over k = l, l+32, ..., k != max),
// with Q their Kogge-Stone total.  Warp per word.
__global__ void __launch_bounds__(256) k_model_lane_q(int V, int Vd, int K, float alpha, const float* __restrict__ phi,
                                                      const uint32_t* __restrict__ top2, float* __restrict__ ql,
                                                      float4* __restrict__ phi4) {
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int w = Vd + blockIdx.x * warps + wid; w < V; w += gridDim.x * warps) {
        const int k1 = (int)(__ldg(top2 + w) & 0xffffu);
        const float* row = phi + (size_t)w * K;
        float acc = 0.0f;
        for (int k = lane; k < K; k += 32)
            if (k != k1) acc = ffma(alpha, __ldg(row + k), acc);
        const float Q = __shfl_sync(FULL, warp_ks_scan(acc, lane), 31);
        ql[(size_t)w * 32 + lane] = acc;
        if (lane == 0) phi4[w].w = Q;
    }
}

// One active request: its tokens sit at [tok_off, tok_off+len) of the pool, its topic counts
// in row slot `slot`, and at step s it runs sweep s - start.  It is sampled in items of
// `item_tokens` tokens, one warp each.
struct FoldReq {
    uint32_t tok_off, len, rid, start, slot, pad0, pad1, pad2;
};

struct FoldArgs {
    int K;
    float alpha, Kalpha;
    uint32_t seed_lo, seed_hi;
    const float* phi;
    const uint32_t* top2;
    const float4* phi4;
    const float* ql;
    const FoldReq* reqs;
    const uint32_t* item_req;  // per item: request index << 16 | item index within the request
    int nitems;
    uint32_t item_tokens;
    uint32_t step;
    uint32_t sweeps;
    const uint32_t* words;
    uint16_t* z;
    uint32_t* rows;     // per slot K entries (k << 16 | count), ascending k
    uint32_t* row_nnz;  // per slot
    float* theta;       // per slot K floats, in pinned host memory
};

__device__ __forceinline__ float foldin_uniform(uint32_t seed_lo, uint32_t seed_hi, uint32_t rid, uint32_t sweep,
                                                uint32_t pos) {
    const uint32_t x = philox_x0(pos, rid, sweep, 0x464F4C44u, seed_lo, seed_hi);
    return u2f(x >> 8) * 0x1p-24f;
}

__device__ __forceinline__ uint32_t foldin_init(uint32_t seed_lo, uint32_t seed_hi, uint32_t rid, uint32_t pos,
                                                int K) {
    const uint32_t x = philox_x0(pos, rid, 0xFFFFFFFFu, 0x46494E49u, seed_lo, seed_hi);
    return (uint32_t)(((unsigned long long)x * (unsigned long long)(uint32_t)K) >> 32);
}

// A word's phi row in the frozen matrix with its max topic zeroed, as a sampler's view of a
// word column.
struct PhiRow {
    const float* __restrict__ prow;
    int mk;
    __device__ __forceinline__ float operator()(int k) const { return k == mk ? 0.0f : __ldg(prow + k); }
};

// The S-bucket draw among lane ls's entries ls, ls + 32, ... of the row (lane_draw with phi
// gathered from the frozen matrix): the first entry with phi > 0 whose partial sum exceeds
// t2, else the last entry with phi > 0, else the max topic.
__device__ __forceinline__ int fold_lane_draw(const uint32_t* __restrict__ row, uint32_t ls, uint32_t nnz,
                                              const PhiRow& phi, float t2) {
    float acc = 0.0f;
    int last = -1;
    for (uint32_t q = ls; q < nnz; q += 128u) {
        uint32_t e[4];
        float c[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = q + 32u * j < nnz ? __ldg(row + q + 32u * j) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = q + 32u * j < nnz ? phi((int)(e[j] >> 16)) : 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (q + 32u * j >= nnz) break;
            acc = ffma(u2f(e[j] & 0xffffu), c[j], acc);
            if (c[j] > 0.0f) {
                last = (int)(e[j] >> 16);
                if (t2 < acc) return last;
            }
        }
    }
    return last >= 0 ? last : phi.mk;
}

// The row's counts of topics k1 and k2 (0 when it has none), by one binary search for both.
__device__ __forceinline__ void row_counts(const uint32_t* __restrict__ row, uint32_t nnz, uint32_t k1, uint32_t k2,
                                           uint32_t& c1, uint32_t& c2) {
    const uint32_t* p1 = row;
    const uint32_t* p2 = row;
    for (uint32_t n = nnz; n > 1u;) {
        const uint32_t h = n >> 1;
        const uint32_t e1 = __ldg(p1 + h), e2 = __ldg(p2 + h);
        if ((e1 >> 16) <= k1) p1 += h;
        if ((e2 >> 16) <= k2) p2 += h;
        n -= h;
    }
    const uint32_t e1 = __ldg(p1), e2 = __ldg(p2);
    c1 = (e1 >> 16) == k1 ? e1 & 0xffffu : 0u;
    c2 = (e2 >> 16) == k2 ? e2 & 0xffffu : 0u;
}

// Q-bucket draws of the tokens in `todo` (words w, max topics mk, rests tt of the targets;
// lane = token) for K <= 1024, where a lane of Q has one round of topics: warp_q_draw for
// four tokens at a time, their loads and scans side by side.  The lane's own token's topic
// goes to znew.
constexpr int kFoldQ = 4;
__device__ __forceinline__ void fold_q_draws(const FoldArgs& a, unsigned todo, uint32_t w, int mk, float tt, int& znew,
                                             int lane) {
    while (todo) {
        int j[kFoldQ], m[kFoldQ], key[kFoldQ];
        const float* prow[kFoldQ];
        float QL[kFoldQ], QP[kFoldQ], t2[kFoldQ], cz[kFoldQ], P[kFoldQ];
        int n = 0;
#pragma unroll
        for (int t = 0; t < kFoldQ; ++t) {
            // past the last token the first is drawn again
            j[t] = t == 0 || todo ? __ffs(todo) - 1 : j[0];
            if (todo) ++n;
            todo &= todo - 1u;
            const uint32_t wj = __shfl_sync(FULL, w, j[t]);
            m[t] = __shfl_sync(FULL, mk, j[t]);
            QL[t] = __ldg(a.ql + (size_t)wj * 32 + lane);
            prow[t] = a.phi + (size_t)wj * a.K;
        }
#pragma unroll
        for (int t = 0; t < kFoldQ; ++t) QP[t] = warp_ks_scan(QL[t], lane);
#pragma unroll
        for (int t = 0; t < kFoldQ; ++t) {
            const float ttj = __shfl_sync(FULL, tt, j[t]);
            const unsigned cand = __ballot_sync(FULL, ttj < QP[t] && QL[t] > 0.0f), pos = __ballot_sync(FULL, QL[t] > 0.0f);
            const int ls = cand ? __ffs(cand) - 1 : (pos ? 31 - __clz(pos) : 0);
            const float prev = __shfl_sync(FULL, QP[t], ls > 0 ? ls - 1 : 0);
            t2[t] = ls > 0 ? fsub(ttj, prev) : ttj;
            key[t] = ls + 32 * lane;
            cz[t] = key[t] < a.K && key[t] != m[t] ? __ldg(prow[t] + key[t]) : 0.0f;
        }
#pragma unroll
        for (int t = 0; t < kFoldQ; ++t) P[t] = warp_ks_scan(fmul(a.alpha, cz[t]), lane);
#pragma unroll
        for (int t = 0; t < kFoldQ; ++t) {
            const unsigned f = __ballot_sync(FULL, cz[t] > 0.0f && t2[t] < P[t]), v = __ballot_sync(FULL, cz[t] > 0.0f);
            const int from = f ? __ffs(f) - 1 : 31 - __clz(v);
            const int z = f || v ? __shfl_sync(FULL, key[t], from) : m[t];
            if (t < n && lane == j[t]) znew = z;
        }
    }
}

// Lane sums of one row against kFoldWords words at a time, into their slots: lane l sums the
// row's entries l, l + 32, ... serially (the training sampler's order), the gathers of all
// words' first NS steps issued before any is used.  c and k hold the lane's first four
// entries (count 0 where the row has none: fmaf(0, phi, acc) is acc, as is the max topic's
// term).
constexpr int kFoldWords = 4;
template <int NS>
__device__ __forceinline__ void fold_rows(const FoldArgs& a, const uint32_t* __restrict__ row, uint32_t nnz,
                                          const float (&c)[4], const uint32_t (&k)[4], const uint2* list, int nrows,
                                          float* slots, int lane) {
    for (int i = 0; i < nrows; i += kFoldWords) {
        const float* prow[kFoldWords];
        uint32_t mk[kFoldWords];
        float v[kFoldWords][NS], acc[kFoldWords];
#pragma unroll
        for (int t = 0; t < kFoldWords; ++t) {
            const uint2 q = list[min(i + t, nrows - 1)];
            prow[t] = a.phi + (size_t)q.x * a.K;
            mk[t] = q.y;
#pragma unroll
            for (int s = 0; s < NS; ++s) v[t][s] = __ldg(prow[t] + k[s]);
        }
#pragma unroll
        for (int t = 0; t < kFoldWords; ++t) {
            acc[t] = 0.0f;
#pragma unroll
            for (int s = 0; s < NS; ++s)
                if (k[s] != mk[t]) acc[t] = ffma(c[s], v[t][s], acc[t]);
        }
        if (NS == 4) {
            for (uint32_t q = 128u; q < nnz; q += 128u) {
                float cc[NS];
                uint32_t kk[NS];
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const uint32_t at = q + 32u * s + (uint32_t)lane;
                    const uint32_t e = at < nnz ? __ldg(row + at) : 0u;
                    cc[s] = u2f(e & 0xffffu);
                    kk[s] = e >> 16;
                }
#pragma unroll
                for (int t = 0; t < kFoldWords; ++t)
#pragma unroll
                    for (int s = 0; s < NS; ++s) v[t][s] = __ldg(prow[t] + kk[s]);
#pragma unroll
                for (int t = 0; t < kFoldWords; ++t)
#pragma unroll
                    for (int s = 0; s < NS; ++s)
                        if (kk[s] != mk[t]) acc[t] = ffma(cc[s], v[t][s], acc[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < kFoldWords; ++t)
            if (i + t < nrows) slots[kSlotWords * (i + t) + lane] = acc[t];
    }
}

// One sweep of every active request: warp per work item, the three parts of the training
// sampler's groups (sample_groups) with every token its own word: the tokens are screened
// thread-per-token, the request's row is summed against each unsettled token's word
// (consecutive tokens of one word share a sum), and each token decides by itself.  What
// bounds it is the latency of the gathers of phi, 4 KB a word at K=1024 from a matrix larger
// than L2: the lane's first four row entries sit in registers for the whole item, and four
// words' gathers of four row steps are in flight together (16 loads; two words: 8.4 against
// 8.1 ms per 2,048 requests, eight at 2 CTAs per SM: 10.6).  A warp takes one item, so that
// the hardware's CTA scheduler balances the items, longest requests first (7.2 -> 6.7 ms).
// With the request's counts and row rebuilt for every item and one word at a time, 2,048
// requests of 30 sweeps took 27.3 ms, one of 900 tokens 1.81 ms (now 6.7 and 0.71).
constexpr int kFoldWarpWords = 32 * kSlotWords + 64;
__global__ void __launch_bounds__(256, 3) k_foldin(FoldArgs a) {
    extern __shared__ float smf[];
    const int warps = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* slots = smf + (size_t)kFoldWarpWords * wid;
    uint2* list = reinterpret_cast<uint2*>(slots + 32 * kSlotWords);
    const int r = blockIdx.x * warps + wid;
    if (r < a.nitems) {
        const uint32_t ir = __ldg(a.item_req + r);
        const FoldReq it = a.reqs[ir >> 16];
        const uint32_t begin = (ir & 0xffffu) * a.item_tokens, end = min(begin + a.item_tokens, it.len);
        const uint32_t sweep = a.step - it.start;
        const uint32_t* row = a.rows + (size_t)it.slot * a.K;
        const uint32_t nnz = __ldg(a.row_nnz + it.slot);
        float c[4];
        uint32_t k[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t e = (uint32_t)lane + 32u * s < nnz ? __ldg(row + lane + 32 * s) : 0u;
            c[s] = u2f(e & 0xffffu);
            k[s] = e >> 16;
        }
        for (uint32_t g = begin; g < end; g += 32) {
            const uint32_t pos = g + lane;
            const bool valid = pos < end;
            uint32_t w = 0;
            int mk = 0;
            float pmax = 0.0f, u = 0.0f, Q = 0.0f;
            bool ea = false;
            if (valid) {
                w = __ldg(a.words + it.tok_off + pos);
                const uint32_t t2 = __ldg(a.top2 + w);
                mk = (int)(t2 & 0xffffu);
                const float4 ph = __ldg(a.phi4 + w);
                uint32_t cmax, c2;
                row_counts(row, nnz, t2 & 0xffffu, t2 >> 16, cmax, c2);
                u = foldin_uniform(a.seed_lo, a.seed_hi, it.rid, sweep, pos);
                pmax = fmul(fadd(u2f(cmax), a.alpha), ph.x);
                const float shat = ffma(u2f(c2), ph.y, fmul(u2f(it.len - cmax - c2), ph.z));
                Q = ph.w;
                ea = fmul(u, fadd(fadd(pmax, shat), Q)) < pmax;
            }
            int znew = mk;
            Draw dr{BR_NONE, 0u, 0.0f, 0.0f};
            const unsigned need = __ballot_sync(FULL, valid && !ea);
            const bool mine = (need >> lane) & 1u;
            const unsigned below = need & ((1u << lane) - 1u);
            const uint32_t wp = __shfl_sync(FULL, w, below ? 31 - __clz(below) : lane);
            const bool lead = mine && (!below || w != wp);
            const unsigned leaders = __ballot_sync(FULL, lead);
            if (need) {
                const int nrows = __popc(leaders);
                const int ri = __popc(leaders & ((2u << lane) - 1u)) - 1;
                if (lead) list[ri] = make_uint2(w, (uint32_t)mk);
                __syncwarp();
                if (nnz > 64u) fold_rows<4>(a, row, nnz, c, k, list, nrows, slots, lane);
                else if (nnz > 32u) fold_rows<2>(a, row, nnz, c, k, list, nrows, slots, lane);
                else fold_rows<1>(a, row, nnz, c, k, list, nrows, slots, lane);
                __syncwarp();
                decide_tokens<false>(slots, mine ? ri : 0, mine, false, pmax, Q, u, lane, dr);
                __syncwarp();  // the slots may be overwritten
            }
            const unsigned qm = __ballot_sync(FULL, dr.kind == BR_Q);
            uint32_t qw = 0xffffffffu;
            float QL = 0.0f, QP = 0.0f;
            if (a.K <= 1024) fold_q_draws(a, qm, w, mk, dr.t, znew, lane);
            else for (unsigned b = qm; b; b &= b - 1u) {
                const int j = __ffs(b) - 1;
                const uint32_t wj = __shfl_sync(FULL, w, j);
                const int mkj = __shfl_sync(FULL, mk, j);
                if (wj != qw) {
                    qw = wj;
                    QL = __ldg(a.ql + (size_t)wj * 32 + lane);
                    QP = warp_ks_scan(QL, lane);
                }
                const float tt = __shfl_sync(FULL, dr.t, j);
                const int zq = warp_q_draw<1>(PhiRow{a.phi + (size_t)wj * a.K, mkj}, tt, QL, QP, a.K, a.alpha, mkj, lane,
                                              nullptr, 0);
                if (lane == j) znew = zq;
            }
            if (dr.kind == BR_S) znew = fold_lane_draw(row, dr.ls, nnz, PhiRow{a.phi + (size_t)w * a.K, mk}, dr.t);
            if (valid) a.z[it.tok_off + pos] = (uint16_t)znew;
        }
    }
}

// The requests' topic counts, CTA per request from `first` on: the row of the next sweep's
// start (of the first sweep's, from the Philox initial topics, with INIT), or after the last
// sweep theta = (n_dk + alpha) / (n_d + K*alpha), written straight to host memory.  Shared
// memory: 16-bit counts (a request has at most 65,535 tokens) and the bitmap of the topics
// that have one.
template <bool INIT>
__global__ void __launch_bounds__(256) k_fold_build(FoldArgs a, int first) {
    extern __shared__ uint32_t smu[];
    __shared__ uint32_t wsum[8];
    const FoldReq q = a.reqs[first + blockIdx.x];
    const int hw = Hist<true>::words(a.K), bw = (a.K + 31) >> 5;
    const Hist<true> hist{smu};
    uint32_t* bits = smu + hw;
    for (int i = threadIdx.x; i < hw + bw; i += blockDim.x) smu[i] = 0u;
    __syncthreads();
    for (uint32_t base = 0; base < q.len; base += 4u * blockDim.x) {
        uint32_t k[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t pos = base + (uint32_t)s * blockDim.x + threadIdx.x;
            k[s] = 0xffffffffu;
            if (pos < q.len) {
                k[s] = INIT ? foldin_init(a.seed_lo, a.seed_hi, q.rid, pos, a.K) : (uint32_t)__ldg(a.z + q.tok_off + pos);
                if (k[s] >= (uint32_t)a.K) k[s] = 0;  // topics are written < K; keep the index in bounds
            }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (k[s] != 0xffffffffu) hist_token(hist, bits, k[s]);
    }
    __syncthreads();
    if (!INIT && a.step - q.start == a.sweeps - 1u) {
        float* th = a.theta + (size_t)q.slot * a.K;
        const float den = fadd(u2f(q.len), a.Kalpha);
        for (int k = threadIdx.x; k < a.K; k += blockDim.x)
            th[k] = __fdiv_rn(fadd(u2f(hist.get((uint32_t)k)), a.alpha), den);
        return;
    }
    uint32_t* out = a.rows + (size_t)q.slot * a.K;
    const uint32_t nnz =
        cta_compact(bw, hist, bits, wsum, [&](uint32_t k, uint32_t h, uint32_t p) { out[p] = (k << 16) | h; });
    if (threadIdx.x == 0) a.row_nnz[q.slot] = nnz;
}

}  // namespace dev
}  // namespace lda

#define CUDA_TRY(expr)                                                                         \
    do {                                                                                       \
        cudaError_t e_ = (expr);                                                               \
        if (e_ != cudaSuccess) {                                                               \
            cudaGetLastError();                                                                \
            return fail(LDA_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_));         \
        }                                                                                      \
    } while (0)

// ------------------------------------------------------------------ model

struct lda_model {
    int device = 0;
    int K = 0;
    int64_t V = 0;
    float alpha = 0, beta = 0;
    float* phi = nullptr;
    uint32_t* top2 = nullptr;
    float4* phi4 = nullptr;
    float* ql = nullptr;
    int64_t bytes = 0;
    ~lda_model() {
        cudaSetDevice(device);
        cudaFree(phi);
        cudaFree(top2);
        cudaFree(phi4);
        cudaFree(ql);
    }
};

extern "C" int lda_model_from_trainer(lda_trainer* t, int64_t device_budget, lda_model** out) {
    if (!t || !out) return fail(LDA_ERR_ARG, "null argument");
    *out = nullptr;
    int rc;
    // counts and word statistics of the trainer's current topics
    if ((rc = lda_update_wt(t)) || (rc = lda_max_topic(t)) || (rc = lda_trainer_sync(t))) return rc;
    std::unique_ptr<lda_model> m(new lda_model());
    ModelSource src;
    if ((rc = trainer_model_source(t, &src))) return rc;
    m->device = src.device;
    m->K = src.K;
    m->V = src.V;
    m->alpha = src.alpha;
    m->beta = src.beta;
    cudaStream_t stream = (cudaStream_t)src.stream;
    const int64_t need = m->V * m->K * 4 + m->V * (4 + 16 + 128);
    if (device_budget > 0 && need > device_budget)
        return fail(LDA_ERR_DEVICE_MEM, "model needs %lld bytes, budget is %lld", (long long)need, (long long)device_budget);
    CUDA_TRY(cudaSetDevice(m->device));
    cudaError_t e = cudaMalloc(&m->phi, sizeof(float) * (size_t)m->V * m->K);
    if (e == cudaSuccess) e = cudaMalloc(&m->top2, sizeof(uint32_t) * (size_t)m->V);
    if (e == cudaSuccess) e = cudaMalloc(&m->phi4, sizeof(float4) * (size_t)m->V);
    if (e == cudaSuccess) e = cudaMalloc(&m->ql, sizeof(float) * 32 * (size_t)m->V);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(LDA_ERR_DEVICE_MEM, "cudaMalloc of the model failed: %s", cudaGetErrorString(e));
    }
    m->bytes = need;
    dev::PhiArgs a;
    a.V = (int)m->V;
    a.Vd = src.Vd;
    a.K = m->K;
    a.beta = m->beta;
    a.Vbeta = (float)m->V * m->beta;
    a.n_k = src.n_k;
    a.dwt = src.dwt;
    a.swt_off = src.swt_off;
    a.swt_nnz = src.swt_nnz;
    a.swt_ent = src.swt_ent;
    a.phi = m->phi;
    const size_t smem = sizeof(float) * (size_t)m->K;
    CUDA_TRY(raise_smem_limit((const void*)dev::k_phi_dense, smem));
    const int grid = (int)std::min<int64_t>(4096, (m->V + 7) / 8);
    dev::k_phi_dense<<<grid, 256, smem, stream>>>(a);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(m->top2, src.top2, sizeof(uint32_t) * (size_t)m->V, cudaMemcpyDeviceToDevice, stream));
    CUDA_TRY(cudaMemcpyAsync(m->phi4, src.phi4, sizeof(float4) * (size_t)m->V, cudaMemcpyDeviceToDevice, stream));
    CUDA_TRY(cudaMemcpyAsync(m->ql, src.ql, sizeof(float) * 32 * (size_t)m->V, cudaMemcpyDeviceToDevice, stream));
    if (m->K > dev::kLargeK && m->V > src.Vd) {
        const int grid = (int)std::min<int64_t>(4096, (m->V - src.Vd + 7) / 8);
        dev::k_model_lane_q<<<grid, 256, 0, stream>>>((int)m->V, src.Vd, m->K, m->alpha, m->phi, m->top2, m->ql,
                                                      reinterpret_cast<float4*>(m->phi4));
        CUDA_TRY(cudaGetLastError());
    }
    CUDA_TRY(cudaStreamSynchronize(stream));
    *out = m.release();
    return LDA_OK;
}

extern "C" int lda_model_info(const lda_model* m, int32_t* K, int64_t* V, int64_t* bytes) {
    if (!m) return fail(LDA_ERR_ARG, "null model");
    if (K) *K = m->K;
    if (V) *V = m->V;
    if (bytes) *bytes = m->bytes;
    return LDA_OK;
}

extern "C" int lda_model_get_phi(const lda_model* m, int32_t w, float* out) {
    if (!m || !out || w < 0 || w >= m->V) return fail(LDA_ERR_ARG, "bad arguments");
    CUDA_TRY(cudaSetDevice(m->device));
    CUDA_TRY(cudaMemcpy(out, m->phi + (size_t)w * m->K, sizeof(float) * m->K, cudaMemcpyDeviceToHost));
    return LDA_OK;
}

extern "C" void lda_model_free(lda_model* m) { delete m; }

// ------------------------------------------------------------------ server

namespace {
using Clock = std::chrono::steady_clock;
double now_s() { return std::chrono::duration<double>(Clock::now().time_since_epoch()).count(); }
constexpr int kRing = 3;      // host item buffers / events
constexpr int kFoldWarps = 8; // most warps per CTA of the fold-in kernel
constexpr int kInFlight = 2;  // steps queued on the stream before the host waits
}  // namespace

struct lda_server {
    lda_model* m = nullptr;
    int device = 0;
    cudaStream_t st = nullptr;
    int sweeps = 30, max_active = 0, num_sms = 0;
    uint32_t item_tokens = 32;
    uint64_t seed = 0;
    int64_t tok_cap = 0, max_items = 0;
    size_t smem_build = 0;
    uint32_t* d_words = nullptr;
    uint16_t* d_z = nullptr;
    uint32_t *d_rows = nullptr, *d_row_nnz = nullptr;  // per slot
    // the active requests' table and the item list behind it, uploaded when the set of active
    // requests has changed
    unsigned char* d_table = nullptr;
    unsigned char* h_table[kRing] = {};
    int64_t table_items = 0;  // of the table on the device
    std::vector<int64_t> item_at;  // scratch of the item list's sort
    bool table_stale = true;
    cudaEvent_t ev[kRing] = {};
    uint32_t* h_words = nullptr;
    float* h_theta = nullptr;
    std::map<int64_t, int64_t> free_iv;  // token pool free intervals: offset -> length
    std::vector<int> free_slots;
    struct Pending {
        uint32_t rid;
        std::vector<uint32_t> words;
        double t_submit;
    };
    struct Active {
        uint32_t rid, len;
        int64_t off;
        uint32_t start;   // the step of its first sweep
        int sweep, slot;  // sweeps issued so far
        double t_submit;
        int64_t last_step;
    };
    struct Done {
        uint32_t rid;
        std::vector<float> theta;
        double t_submit, t_done;
    };
    std::deque<Pending> queue;
    std::vector<Active> active;
    std::deque<Active> finishing;      // last sweep issued, waiting for its step's event
    std::deque<int64_t> inflight;      // issued steps not yet collected
    std::deque<Done> done;
    int64_t steps = 0, kernel_launches = 0;

    ~lda_server() {
        cudaSetDevice(device);
        if (st) cudaStreamSynchronize(st);
        cudaFree(d_words);
        cudaFree(d_z);
        cudaFree(d_rows);
        cudaFree(d_row_nnz);
        cudaFree(d_table);
        for (int i = 0; i < kRing; ++i) {
            cudaFreeHost(h_table[i]);
            if (ev[i]) cudaEventDestroy(ev[i]);
        }
        cudaFreeHost(h_words);
        cudaFreeHost(h_theta);
        if (st) cudaStreamDestroy(st);
    }

    size_t table_bytes(int64_t items) const {
        return sizeof(dev::FoldReq) * (size_t)max_active + sizeof(uint32_t) * (size_t)items;
    }

    bool alloc_tokens(int64_t len, int64_t* off) {
        for (auto it = free_iv.begin(); it != free_iv.end(); ++it) {
            if (it->second >= len) {
                *off = it->first;
                const int64_t rest = it->second - len, noff = it->first + len;
                free_iv.erase(it);
                if (rest > 0) free_iv[noff] = rest;
                return true;
            }
        }
        return false;
    }

    void free_tokens(int64_t off, int64_t len) {
        auto it = free_iv.emplace(off, len).first;
        auto nx = std::next(it);
        if (nx != free_iv.end() && it->first + it->second == nx->first) {
            it->second += nx->second;
            free_iv.erase(nx);
        }
        if (it != free_iv.begin()) {
            auto pv = std::prev(it);
            if (pv->first + pv->second == it->first) {
                pv->second += it->second;
                free_iv.erase(it);
            }
        }
    }

    // Retires the requests whose last step is `step` (its event has completed).
    void retire_through(int64_t step, double t) {
        while (!finishing.empty() && finishing.front().last_step <= step) {
            const Active& a = finishing.front();
            Done d;
            d.rid = a.rid;
            d.theta.assign(h_theta + (size_t)a.slot * m->K, h_theta + (size_t)(a.slot + 1) * m->K);
            d.t_submit = a.t_submit;
            d.t_done = t;
            done.push_back(std::move(d));
            free_tokens(a.off, a.len);
            free_slots.push_back(a.slot);
            finishing.pop_front();
        }
    }

    // Collects completed steps: blocking on the oldest while more than `keep` are queued,
    // then every step whose event has already completed.  Returns requests retired.
    int collect(size_t keep, int* rc) {
        const size_t before = done.size();
        while (!inflight.empty()) {
            const int64_t k = inflight.front();
            cudaEvent_t e = ev[k % kRing];
            if (inflight.size() > keep) {
                const cudaError_t err = cudaEventSynchronize(e);
                if (err != cudaSuccess) {
                    cudaGetLastError();
                    *rc = fail(LDA_ERR_CUDA, "fold-in step failed: %s", cudaGetErrorString(err));
                    return 0;
                }
            } else {
                const cudaError_t q = cudaEventQuery(e);
                if (q == cudaErrorNotReady) break;
                if (q != cudaSuccess) {
                    cudaGetLastError();
                    *rc = fail(LDA_ERR_CUDA, "fold-in step failed: %s", cudaGetErrorString(q));
                    return 0;
                }
            }
            inflight.pop_front();
            retire_through(k, now_s());
        }
        return (int)(done.size() - before);
    }
};

extern "C" int lda_server_create(lda_model* m, int64_t max_tokens, int32_t max_active, int32_t sweeps, uint64_t seed,
                                 lda_server** out) {
    if (!m || !out) return fail(LDA_ERR_ARG, "null argument");
    *out = nullptr;
    if (sweeps < 1 || max_active < 1 || max_tokens < 0) return fail(LDA_ERR_ARG, "sweeps and max_active must be >= 1");
    if (max_tokens > ((int64_t)1 << 31)) return fail(LDA_ERR_ARG, "token pool above 2^31 tokens");
    if (max_active > 65535) return fail(LDA_ERR_ARG, "max_active above 65535");
    std::unique_ptr<lda_server> s(new lda_server());
    s->m = m;
    s->device = m->device;
    s->sweeps = sweeps;
    s->max_active = max_active;
    s->seed = seed;
    CUDA_TRY(cudaSetDevice(s->device));
    if (max_tokens == 0) {
        // admission by free HBM: the token pool (4 B word + 2 B topic per token) holds one
        // token per 8 bytes of a quarter of the free device memory
        size_t fr = 0, tot = 0;
        CUDA_TRY(cudaMemGetInfo(&fr, &tot));
        max_tokens = std::min<int64_t>((int64_t)(fr / 4) / 8, (int64_t)1 << 30);
    }
    s->tok_cap = max_tokens;
    s->max_items = (int64_t)max_active + max_tokens / s->item_tokens + 1;
    cudaError_t e = cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&s->d_words, sizeof(uint32_t) * (size_t)max_tokens);
    if (e == cudaSuccess) e = cudaMalloc(&s->d_z, sizeof(uint16_t) * (size_t)max_tokens);
    if (e == cudaSuccess) e = cudaMalloc(&s->d_rows, sizeof(uint32_t) * (size_t)max_active * m->K);
    if (e == cudaSuccess) e = cudaMalloc(&s->d_row_nnz, sizeof(uint32_t) * (size_t)max_active);
    if (e == cudaSuccess) e = cudaMalloc(&s->d_table, s->table_bytes(s->max_items));
    for (int i = 0; i < kRing && e == cudaSuccess; ++i) {
        e = cudaMallocHost(&s->h_table[i], s->table_bytes(s->max_items));
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->ev[i], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaMallocHost(&s->h_words, sizeof(uint32_t) * (size_t)max_tokens);
    if (e == cudaSuccess) e = cudaMallocHost(&s->h_theta, sizeof(float) * (size_t)max_active * m->K);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(LDA_ERR_DEVICE_MEM, "server allocation failed: %s", cudaGetErrorString(e));
    }
    s->free_iv[0] = max_tokens;
    for (int i = max_active - 1; i >= 0; --i) s->free_slots.push_back(i);
    int max_smem = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device));
    CUDA_TRY(cudaDeviceGetAttribute(&s->num_sms, cudaDevAttrMultiProcessorCount, s->device));
    s->smem_build = ((size_t)dev::Hist<true>::words(m->K) + (size_t)(m->K + 31) / 32) * 4;
    if (s->smem_build > (size_t)max_smem) return fail(LDA_ERR_ARG, "K=%d does not fit in shared memory", m->K);
    CUDA_TRY(raise_smem_limit((const void*)dev::k_fold_build<true>, s->smem_build));
    CUDA_TRY(raise_smem_limit((const void*)dev::k_fold_build<false>, s->smem_build));
    CUDA_TRY(raise_smem_limit((const void*)dev::k_foldin, sizeof(float) * dev::kFoldWarpWords * kFoldWarps));
    CUDA_TRY(cudaStreamSynchronize(s->st));
    *out = s.release();
    return LDA_OK;
}

extern "C" int lda_server_destroy(lda_server* s) {
    delete s;
    return LDA_OK;
}

extern "C" int lda_server_set_item_tokens(lda_server* s, int32_t n) {
    if (!s || n < 32 || n % 32) return fail(LDA_ERR_ARG, "item size must be a positive multiple of 32");
    if (!s->active.empty() || !s->inflight.empty()) return fail(LDA_ERR_STATE, "server is busy");
    const int64_t need = (int64_t)s->max_active + s->tok_cap / n + 1;
    if (need > s->max_items) {
        CUDA_TRY(cudaSetDevice(s->device));
        CUDA_TRY(cudaStreamSynchronize(s->st));
        cudaFree(s->d_table);
        s->d_table = nullptr;
        for (int i = 0; i < kRing; ++i) {
            cudaFreeHost(s->h_table[i]);
            s->h_table[i] = nullptr;
        }
        s->max_items = 0;
        s->table_stale = true;
        cudaError_t e = cudaMalloc(&s->d_table, s->table_bytes(need));
        for (int i = 0; i < kRing && e == cudaSuccess; ++i) e = cudaMallocHost(&s->h_table[i], s->table_bytes(need));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(LDA_ERR_DEVICE_MEM, "item table allocation failed: %s", cudaGetErrorString(e));
        }
        s->max_items = need;
    }
    s->item_tokens = (uint32_t)n;
    return LDA_OK;
}

extern "C" int lda_server_submit(lda_server* s, uint32_t rid, const int32_t* words, int32_t len) {
    if (!s || !words) return fail(LDA_ERR_ARG, "null argument");
    if (len < 1 || len > 65535) return fail(LDA_ERR_ARG, "request length %d outside [1, 65535]", len);
    if (len > s->tok_cap)
        return fail(LDA_ERR_DEVICE_MEM, "request of %d tokens exceeds the token pool (%lld)", len, (long long)s->tok_cap);
    lda_server::Pending p;
    p.rid = rid;
    p.t_submit = now_s();
    p.words.resize(len);
    for (int32_t i = 0; i < len; ++i) {
        if (words[i] < 0 || words[i] >= s->m->V)
            return fail(LDA_ERR_ARG, "word %d of request %u outside the vocabulary", words[i], rid);
        p.words[i] = (uint32_t)words[i];
    }
    s->queue.push_back(std::move(p));
    return LDA_OK;
}

// Issues one step: admits queued requests that fit (FIFO, by token pool and slots), queues
// one sweep of every active request on the stream, and moves requests whose last sweep it
// is to the finishing list.  Completion is collected by lda_server::collect.
static int server_issue(lda_server* s) {
    CUDA_TRY(cudaSetDevice(s->device));
    int rc = LDA_OK;
    // the host buffers of step `steps` were last used by step `steps - kRing`
    s->collect(kInFlight - 1, &rc);
    if (rc) return rc;
    const int64_t k = s->steps;
    const int nold = (int)s->active.size();
    // new requests' words go up in one copy per run of neighbouring pool ranges
    int64_t run0 = 0, run1 = 0;
    auto upload = [&]() -> int {
        if (run1 > run0)
            CUDA_TRY(cudaMemcpyAsync(s->d_words + run0, s->h_words + run0, sizeof(uint32_t) * (size_t)(run1 - run0),
                                     cudaMemcpyHostToDevice, s->st));
        return LDA_OK;
    };
    while (!s->queue.empty() && (int)s->active.size() < s->max_active && !s->free_slots.empty()) {
        auto& p = s->queue.front();
        int64_t off;
        if (!s->alloc_tokens((int64_t)p.words.size(), &off)) break;
        lda_server::Active a;
        a.rid = p.rid;
        a.len = (uint32_t)p.words.size();
        a.off = off;
        a.sweep = 0;
        a.start = (uint32_t)k;
        a.slot = s->free_slots.back();
        s->free_slots.pop_back();
        a.t_submit = p.t_submit;
        a.last_step = -1;
        std::memcpy(s->h_words + off, p.words.data(), sizeof(uint32_t) * a.len);
        if (off != run1) {
            if ((rc = upload())) return rc;
            run0 = off;
        }
        run1 = off + a.len;
        s->active.push_back(a);
        s->queue.pop_front();
        s->table_stale = true;
    }
    if ((rc = upload())) return rc;
    if (s->active.empty()) return LDA_OK;
    if (s->max_items == 0) return fail(LDA_ERR_STATE, "the server has no item table (a failed resize)");
    const uint32_t T = s->item_tokens;
    const int nreq = (int)s->active.size();
    if (s->table_stale) {
        dev::FoldReq* reqs = reinterpret_cast<dev::FoldReq*>(s->h_table[k % kRing]);
        uint32_t* items = reinterpret_cast<uint32_t*>(reqs + nreq);
        // the longest requests' items first (their rows are the longest): a counting sort of
        // the requests by their items
        int64_t n = 0;
        std::vector<int64_t>& at = s->item_at;
        at.assign((65535 + T - 1) / T + 1, 0);
        for (int r = 0; r < nreq; ++r) {
            const auto& a = s->active[r];
            reqs[r] = dev::FoldReq{(uint32_t)a.off, a.len, a.rid, a.start, (uint32_t)a.slot, 0u, 0u, 0u};
            at[(a.len + T - 1) / T] += (a.len + T - 1) / T;
        }
        for (size_t b = at.size(); b-- > 0;) {
            const int64_t c = at[b];
            at[b] = n;
            n += c;
        }
        for (int r = 0; r < nreq; ++r) {
            const uint32_t nitems = (s->active[r].len + T - 1) / T, tag = (uint32_t)r << 16;
            uint32_t* out = items + at[nitems];
            for (uint32_t j = 0; j < nitems; ++j) out[j] = tag | j;
            at[nitems] += nitems;
        }
        CUDA_TRY(cudaMemcpyAsync(s->d_table, reqs, sizeof(dev::FoldReq) * (size_t)nreq + sizeof(uint32_t) * (size_t)n,
                                 cudaMemcpyHostToDevice, s->st));
        s->table_items = n;
        s->table_stale = false;
    }
    const int64_t n = s->table_items;
    dev::FoldArgs fa;
    fa.K = s->m->K;
    fa.alpha = s->m->alpha;
    fa.Kalpha = (float)s->m->K * s->m->alpha;
    fa.seed_lo = (uint32_t)s->seed;
    fa.seed_hi = (uint32_t)(s->seed >> 32);
    fa.phi = s->m->phi;
    fa.top2 = s->m->top2;
    fa.phi4 = s->m->phi4;
    fa.ql = s->m->ql;
    fa.reqs = reinterpret_cast<const dev::FoldReq*>(s->d_table);
    fa.item_req = reinterpret_cast<const uint32_t*>(fa.reqs + nreq);
    fa.nitems = (int)n;
    fa.item_tokens = T;
    fa.step = (uint32_t)k;
    fa.sweeps = (uint32_t)s->sweeps;
    fa.words = s->d_words;
    fa.z = s->d_z;
    fa.rows = s->d_rows;
    fa.row_nnz = s->d_row_nnz;
    fa.theta = s->h_theta;
    if (nreq > nold) {
        dev::k_fold_build<true><<<nreq - nold, 256, s->smem_build, s->st>>>(fa, nold);
        CUDA_TRY(cudaGetLastError());
    }
    // few items: one or a few warps per CTA, so that they spread over the SMs
    const int warps = (int)std::max<int64_t>(1, std::min<int64_t>(kFoldWarps, (n + s->num_sms - 1) / s->num_sms));
    dev::k_foldin<<<(int)((n + warps - 1) / warps), 32 * warps, sizeof(float) * dev::kFoldWarpWords * warps, s->st>>>(fa);
    CUDA_TRY(cudaGetLastError());
    s->kernel_launches++;
    dev::k_fold_build<false><<<nreq, 256, s->smem_build, s->st>>>(fa, 0);
    CUDA_TRY(cudaGetLastError());
    size_t kept = 0;
    for (auto& a : s->active) {
        if (a.sweep++ == s->sweeps - 1) {
            a.last_step = k;
            s->finishing.push_back(a);
        } else {
            s->active[kept++] = a;
        }
    }
    if (kept < s->active.size()) {
        s->active.resize(kept);
        s->table_stale = true;
    }
    CUDA_TRY(cudaEventRecord(s->ev[k % kRing], s->st));
    s->inflight.push_back(k);
    s->steps++;
    return LDA_OK;
}

extern "C" int lda_server_step(lda_server* s, int32_t* n_done) {
    if (!s) return fail(LDA_ERR_ARG, "null server");
    const size_t before = s->done.size();
    int rc;
    if (!s->queue.empty() || !s->active.empty()) {
        if ((rc = server_issue(s))) return rc;
        rc = LDA_OK;
        s->collect(kInFlight, &rc);
    } else {
        rc = LDA_OK;
        s->collect(0, &rc);  // nothing left to issue: wait for the queued steps
    }
    if (rc) return rc;
    if (n_done) *n_done = (int32_t)(s->done.size() - before);
    return LDA_OK;
}

extern "C" int lda_server_poll(lda_server* s, uint32_t* rid, float* theta, double* latency_s) {
    if (!s || !rid) return fail(LDA_ERR_ARG, "null argument");
    if (s->done.empty()) return 0;
    auto& d = s->done.front();
    *rid = d.rid;
    if (theta) std::memcpy(theta, d.theta.data(), sizeof(float) * d.theta.size());
    if (latency_s) *latency_s = d.t_done - d.t_submit;
    s->done.pop_front();
    return 1;
}

extern "C" int lda_server_status(const lda_server* s, int32_t* queued, int32_t* active, int64_t* free_tokens) {
    if (!s) return fail(LDA_ERR_ARG, "null server");
    if (queued) *queued = (int32_t)s->queue.size();
    if (active) *active = (int32_t)(s->active.size() + s->finishing.size());
    if (free_tokens) {
        int64_t f = 0;
        for (auto& kv : s->free_iv) f += kv.second;
        *free_tokens = f;
    }
    return LDA_OK;
}

extern "C" int lda_server_get_topics(lda_server* s, uint32_t rid, uint16_t* out, int32_t len) {
    if (!s || !out) return fail(LDA_ERR_ARG, "null argument");
    for (auto& a : s->active)
        if (a.rid == rid) {
            if ((int32_t)a.len != len) return fail(LDA_ERR_ARG, "request %u has %u tokens", rid, a.len);
            if (a.sweep == 0) return fail(LDA_ERR_STATE, "request %u has not run a sweep yet", rid);
            CUDA_TRY(cudaSetDevice(s->device));
            CUDA_TRY(cudaStreamSynchronize(s->st));
            CUDA_TRY(cudaMemcpy(out, s->d_z + a.off, sizeof(uint16_t) * a.len, cudaMemcpyDeviceToHost));
            return LDA_OK;
        }
    return fail(LDA_ERR_STATE, "request %u is not active", rid);
}

extern "C" int lda_server_stats(const lda_server* s, int64_t* steps, int64_t* kernel_launches) {
    if (!s) return fail(LDA_ERR_ARG, "null server");
    if (steps) *steps = s->steps;
    if (kernel_launches) *kernel_launches = s->kernel_launches;
    return LDA_OK;
}

// Real-time replay of an arrival schedule on an idle server.
extern "C" int lda_serve_replay(lda_server* s, int32_t n, const int64_t* doc_off, const int32_t* words,
                                const double* arrival_s, double* latency_s, float* theta, double* wall_s) {
    if (!s || !doc_off || !words || !arrival_s || !latency_s || n < 0) return fail(LDA_ERR_ARG, "null argument");
    for (int32_t i = 1; i < n; ++i)
        if (arrival_s[i] < arrival_s[i - 1]) return fail(LDA_ERR_ARG, "arrival times must be non-decreasing");
    if (!s->queue.empty() || !s->active.empty() || !s->finishing.empty() || !s->done.empty())
        return fail(LDA_ERR_STATE, "replay needs an idle server (nothing queued, active or unpolled)");
    const double t0 = now_s();
    int32_t next = 0, finished = 0;
    int rc;
    while (finished < n) {
        const double now = now_s() - t0;
        while (next < n && arrival_s[next] <= now) {
            if ((rc = lda_server_submit(s, (uint32_t)next, words + doc_off[next],
                                        (int32_t)(doc_off[next + 1] - doc_off[next]))))
                return rc;
            s->queue.back().t_submit = t0 + arrival_s[next];  // latency counts from the scheduled arrival
            ++next;
        }
        if (s->queue.empty() && s->active.empty()) {
            rc = LDA_OK;
            if (!s->inflight.empty()) {
                s->collect(s->inflight.size() - 1, &rc);  // wait for the oldest queued step
                if (rc) return rc;
            } else if (next < n) {
                const double wait = arrival_s[next] - (now_s() - t0);
                if (wait > 2e-4) std::this_thread::sleep_for(std::chrono::duration<double>(wait - 1e-4));
            }
        } else {
            if ((rc = server_issue(s))) return rc;
            rc = LDA_OK;
            s->collect(kInFlight, &rc);
            if (rc) return rc;
        }
        while (!s->done.empty()) {
            auto& d = s->done.front();
            if (d.rid < (uint32_t)n) {
                if (theta) std::memcpy(theta + (size_t)d.rid * s->m->K, d.theta.data(), sizeof(float) * s->m->K);
                latency_s[d.rid] = d.t_done - d.t_submit;
                ++finished;
            }
            s->done.pop_front();
        }
    }
    if (wall_s) *wall_s = now_s() - t0;
    return LDA_OK;
}
