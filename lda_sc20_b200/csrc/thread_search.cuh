// thread_search.cuh -- the sampler's searches by a single thread: the lane, topic or table place
// whose prefix first exceeds a target, for draws that run thread per token.
//
// The whole warp's draws compare a target with every prefix and take the first above it.  A
// thread's binary search looks at a few of them.  Rounding can leave neighbouring prefixes out of
// order, so each search also says whether its answer is sure to be the first; a token that is not
// sure is drawn by the whole warp.  The header names no CUDA runtime type of its own, so that a
// host compiler with stand-ins for fadd, fmul, fsub, fadd2 and __ldg compiles it too.
#pragma once

namespace lda {
namespace dev {

// How far above the prefix before it a target must be for a sure answer.  Lane prefixes: a
// prefix of a 32-value Kogge-Stone scan is within (1 + 2^-24)^5 of its exact sum.  The smoothing
// table: its entries are out of order by less than 16 units of 2^-24 (thread_split_draw).
constexpr float kPrefixUp = 1.0f + 0x1p-19f;
constexpr float kTableUp = 1.0f + 0x1p-20f;

// Up to this many topics Q-bucket draws run thread per token (QB 0, thread_q_draw).
constexpr int kThreadQTopics = 256;
// Most topics for which a Q-bucket draw's second level is a thread's own search: a lane of Q
// then has at most kThreadQ topics.  (A warp's draw takes 85 warp instructions per token, a
// thread's about 130 per group, and a fifth of the draws are from Q at these sizes; with 32
// topics per lane the thread's search costs as much as four tokens' draws by the warp.)
constexpr int kThreadQ = kThreadQTopics / 32;

// The Kogge-Stone scan of N (even) values held by one thread: element l adds element l - off
// at each step off = 1, 2, ..., the additions of warp_ks_scan's first N lanes, from step 2 on
// two at a time.
template <int N>
__device__ __forceinline__ void thread_ks_scan(float (&v)[N]) {
#pragma unroll
    for (int l = N - 1; l >= 1; --l) v[l] = fadd(v[l], v[l - 1]);
#pragma unroll
    for (int off = 2; off < N; off <<= 1) {
#pragma unroll
        for (int l = N - 2; l >= off; l -= 2) fadd2(v[l], v[l + 1], v[l - off], v[l - off + 1]);
    }
}

// The crossing of t in 32 Kogge-Stone prefixes of non-negative terms held by one thread: a
// binary search with the prefixes halved in registers.  idx is a place with
// v[idx - 1] <= t (prev) and, when any prefix exceeds t, t < v[idx] (at).  Rounding can leave
// the prefixes out of order by a few units in the last place: a prefix is within (1 + 2^-24)^5
// of its exact sum and the exact sums ascend, so when t >= prev (1 + 2^-19) no earlier prefix
// exceeds t, and idx is the first place that does.  `sure` says so (false also when no
// prefix exceeds t).
__device__ __forceinline__ void thread_crossing(const float (&v)[32], float t, int& idx, float& prev, bool& sure) {
    float w[16];
    prev = 0.0f;
    bool up = !(t < v[15]);
    idx = up ? 16 : 0;
    if (up) prev = v[15];
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = up ? v[16 + i] : v[i];
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        up = !(t < w[h - 1]);
        idx += up ? h : 0;
        if (up) prev = w[h - 1];
#pragma unroll
        for (int i = 0; i < h; ++i) w[i] = up ? w[h + i] : w[i];
    }
    sure = t < w[0] && !(t < fmul(prev, kPrefixUp));
}

// Q-bucket draws of all of a group's tokens with `act` (rest tt of the target each), thread
// per token, for K <= 32 kThreadQ: the draws of warp_q_draw.  qps holds the word's 32 Q
// prefixes, qpos the lanes with a positive partial.  `unsure` gets the tokens whose lane the
// search could not be sure of (as thread_crossing).
template <class View>
__device__ __forceinline__ int thread_q_draw(const View& colz, const float* qps, unsigned qpos, float tt, int K,
                                             float alpha, int maxK, bool& unsure) {
    int ls = 0;
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1)
        if (!(tt < qps[ls + h - 1])) ls += h;
    // ls in 0..31: lane 31 is not probed, it is the answer when no other lane exceeds tt
    const float prev = ls > 0 ? qps[ls - 1] : 0.0f;
    unsure = !(tt < qps[ls]) || tt < fmul(prev, kPrefixUp) || !((qpos >> ls) & 1u);
    const float t2 = ls > 0 ? fsub(tt, prev) : tt;
    float cz[kThreadQ], v[kThreadQ];
#pragma unroll
    for (int i = 0; i < kThreadQ; ++i) {
        const int k = ls + 32 * i;
        cz[i] = k < K ? colz(k) : 0.0f;
        v[i] = fmul(alpha, cz[i]);
    }
    thread_ks_scan(v);
    int first = -1, last = -1;
#pragma unroll
    for (int i = kThreadQ - 1; i >= 0; --i) {
        const bool ok = cz[i] > 0.0f;
        if (ok && t2 < v[i]) first = i;
        if (ok && last < 0) last = i;
    }
    const int i = first >= 0 ? first : last;
    return i >= 0 ? ls + 32 * i : maxK;
}

// Q-bucket draws above kThreadQTopics with the word's Q-round table (tab, `qrounds` pairs per
// lane slot), thread per token: the lane, then the first round whose threshold exceeds the
// rest of the target, then the crossing among that round's 32 topics, as warp_q_draw finds
// them; `unsure` as thread_q_draw.
template <class View>
__device__ __forceinline__ int thread_q_draw_table(const View& colz, const float* qps, unsigned qpos, float tt, int K,
                                                   float alpha, const float2* tab, int qrounds, bool& unsure) {
    int ls = 0;
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1)
        if (!(tt < qps[ls + h - 1])) ls += h;
    float prev = ls > 0 ? qps[ls - 1] : 0.0f;
    unsure = !(tt < qps[ls]) || tt < fmul(prev, kPrefixUp) || !((qpos >> ls) & 1u);
    const float t2 = ls > 0 ? fsub(tt, prev) : tt;
    const int n = (K - ls + 31) / 32;  // the lane slot's topics
    const float2* row = tab + ls * qrounds;
    int r = 0;
    float carry = 0.0f;
    for (;; ++r) {
        if (32 * r >= n) {
            unsure = true;
            return 0;
        }
        const float2 e = row[r];
        if (t2 < e.y) {
            carry = e.x;
            break;
        }
    }
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 32 * r + i < n ? fmul(alpha, colz(ls + 32 * (32 * r + i))) : 0.0f;
    thread_ks_scan(v);
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = fadd(carry, v[i]);
    int i;
    bool sure;
    thread_crossing(v, t2, i, prev, sure);
    const int k = ls + 32 * (32 * r + i);
    unsure = unsure || !sure || 32 * r + i >= n || !(colz(min(k, K - 1)) > 0.0f);
    return k;
}

// split_q_draw thread per token (t, and whether to draw, differ by lane; q is a SplitQ), with binary
// searches in the word's prefixes and in T (its round ends first).  The searches compare
// fewer places than split_q_draw's; places may be out of order by rounding, a prefix by
// (1 + 2^-24)^5 (thread_crossing) and T's entries by less than 16 units of 2^-24 (a round's
// prefixes as any, and each carry is at least every sum it is formed from but for that), so
// a target that close to a neighbour is `unsure` and left to split_q_draw.  So is a draw from
// the word's own topics when they take more than one round.
template <class Split>
__device__ __forceinline__ int thread_split_draw(const Split& q, float t, int maxK, int K, float alpha, float beta,
                                                 bool& unsure) {
    unsure = false;
    if (t < q.Qw) {
        if (!q.wp) {
            unsure = true;
            return maxK;
        }
        int e = 0;
#pragma unroll
        for (int h = 16; h >= 1; h >>= 1)
            if (!(t < q.wp[e + h - 1])) e += h;
        unsure = !(t < q.wp[e]) || !((q.wok >> e) & 1u) || (e > 0 && t < fmul(q.wp[e - 1], kPrefixUp));
        return (int)(__ldg(q.ent + min((uint32_t)e, q.nnz - 1u)) >> 16);
    }
    const float t1 = fsub(t, q.Qw);
    const bool left = maxK > 0 && t1 < __ldg(q.T + maxK - 1);
    const float x = left ? t1 : fadd(t1, fmul(alpha, fmul(beta, q.rk(maxK))));
    const int start = left ? 0 : maxK + 1;
    int lo = 0, hi = (K + 31) >> 5;
    const int rounds = hi;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (x < q.tend[mid]) hi = mid; else lo = mid + 1;
    }
    if (lo == rounds) {
        unsure = true;
        return maxK;
    }
    hi = min(K, 32 * lo + 32) - 1;  // x < T[hi], the round's end
    lo = 32 * lo;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (x < __ldg(q.T + mid)) hi = mid; else lo = mid + 1;
    }
    const int k = max(lo, start);
    if (k >= K) {
        unsure = true;
        return maxK;
    }
    unsure = !(fmul(x, kTableUp) < __ldg(q.T + k)) ||
             (k > start && x < fmul(__ldg(q.T + k - 1), kTableUp));
    return k;
}

}  // namespace dev
}  // namespace lda
