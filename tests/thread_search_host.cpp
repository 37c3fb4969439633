// The sampler's searches by a single thread (csrc/thread_search.cuh), compiled for the host with
// IEEE operations in place of the CUDA intrinsics, over arrays of targets.
#include <algorithm>
#include <cstdint>

#define __device__
#define __forceinline__ inline
struct float2 {
    float x, y;
};
template <class T>
static inline T __ldg(const T* p) {
    return *p;
}
namespace lda {
namespace dev {
using std::max;
using std::min;
static inline float fadd(float a, float b) { return a + b; }
static inline float fsub(float a, float b) { return a - b; }
static inline float fmul(float a, float b) { return a * b; }
static inline void fadd2(float& a0, float& a1, float b0, float b1) {
    a0 = a0 + b0;
    a1 = a1 + b1;
}
}  // namespace dev
}  // namespace lda
#include "thread_search.cuh"
using namespace lda::dev;

struct Column {
    const float* col;
    float operator()(int k) const { return col[k]; }
};
struct Split {
    const uint32_t* ent;
    uint32_t nnz;
    float Qw;
    const float *T, *r, *wp;
    unsigned wok;
    const float* tend;
    float rk(int k) const { return r[k]; }
};

extern "C" {
void crossing(int n, const float* terms, const float* t, int* idx, float* prev, uint8_t* sure) {
    for (int i = 0; i < n; ++i) {
        float v[32];
        std::copy(terms + 32 * i, terms + 32 * i + 32, v);
        thread_ks_scan(v);
        bool s;
        thread_crossing(v, t[i], idx[i], prev[i], s);
        sure[i] = s;
    }
}
void q_draw(int n, int K, const float* col, float alpha, int maxK, const float* qps, unsigned qpos, const float* t, int* z,
            uint8_t* unsure) {
    for (int i = 0; i < n; ++i) {
        bool u;
        z[i] = thread_q_draw(Column{col}, qps, qpos, t[i], K, alpha, maxK, u);
        unsure[i] = u;
    }
}
void q_draw_table(int n, int K, const float* col, float alpha, const float* qps, unsigned qpos, const float* tab, int rounds,
                  const float* t, int* z, uint8_t* unsure) {
    for (int i = 0; i < n; ++i) {
        bool u;
        z[i] = thread_q_draw_table(Column{col}, qps, qpos, t[i], K, alpha, (const float2*)tab, rounds, u);
        unsure[i] = u;
    }
}
void split_draw(int n, int K, float alpha, float beta, int maxK, const uint32_t* ent, unsigned nnz, float Qw, const float* T,
                const float* r, const float* wp, unsigned wok, const float* tend, const float* t, int* z, uint8_t* unsure) {
    const Split q{ent, nnz, Qw, T, r, wp, wok, tend};
    for (int i = 0; i < n; ++i) {
        bool u;
        z[i] = thread_split_draw(q, t[i], maxK, K, alpha, beta, u);
        unsure[i] = u;
    }
}
}
