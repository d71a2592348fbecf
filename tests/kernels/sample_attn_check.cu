// sample_attn_kernel alone against 64 bits: random queries and caches, prompt pages shared, later pages a sample's own.
//   sample_attn_check CACHE(f16|bf16) HD KV_HEADS GQA SAMPLES PROMPT OWN PAGE_TOKENS SMS
// prints the relative error (2-norm) over all samples and heads, and the cut it was launched with.  SMS: what sa_split is told (fewer: longer slices).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "sample_attn.cuh"

using namespace cd;

template <class T> T* on_device(const std::vector<T>& v) {
    T* p = nullptr;
    if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess || cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) exit(2);
    return p;
}

template <class KT, int HD> int check(int kv, int gqa, int ns, int prompt, int own, int pt, int sms) {
    const int pps = (prompt + own + pt - 1) / pt, heads = kv * gqa, len = prompt + own, shared = prompt / pt * pt, nsplit = std::min(32, pps);
    std::mt19937_64 gen(7);
    std::normal_distribution<float> normal;
    const size_t page = (size_t)2 * kv * pt * HD, rows = (size_t)ns * heads;
    std::vector<KT> pool((size_t)ns * pps * page);
    std::vector<double> exact(pool.size());
    for (size_t i = 0; i < pool.size(); ++i) {
        pool[i] = KT(normal(gen));
        exact[i] = (double)float(pool[i]);
    }
    std::vector<float> q(rows * HD);
    for (float& x : q) x = 2.0f * normal(gen);
    std::vector<int> table((size_t)ns * pps);
    for (int s = 0; s < ns; ++s)
        for (int j = 0; j < pps; ++j) table[(size_t)s * pps + j] = (s == 0 || (j + 1) * pt <= prompt) ? j : s * pps + j;
    DevState st = {};
    st.pos = len - 1;
    const SaBlocks blocks{gqa, ns};
    const SaSplit cut = sa_split(shared, len, blocks, kv, nsplit, sms);
    if (cut.shared + cut.own > nsplit) return printf("%d slices do not fit %d\n", cut.shared + cut.own, nsplit), 1;
    const float* dq = on_device(q);
    const KT* dpool = on_device(pool);
    float* acc = on_device(std::vector<float>(rows * nsplit * HD));
    float* ml = on_device(std::vector<float>(rows * nsplit * 2));
    unsigned* counters = on_device(std::vector<unsigned>((size_t)blocks.count() * kv));
    __half *hi = on_device(std::vector<__half>(rows * HD)), *lo = on_device(std::vector<__half>(rows * HD));
    const SampleAttn at{dq, on_device(table), on_device(std::vector<DevState>{st}), acc, ml, counters, kv, pt, pps, nsplit, shared, blocks, cut, 1.0f / std::sqrt((float)HD)};
    for (int twice = 0; twice < 2; ++twice)  // (the counters are zero again behind a launch)
        sample_attn_kernel<KT, __half, HD><<<dim3(kv, cut.shared + cut.own, blocks.count()), SA_THREADS>>>(at, dpool, hi, lo);
    std::vector<__half> h(rows * HD), l(rows * HD);
    cudaMemcpy(h.data(), hi, h.size() * 2, cudaMemcpyDeviceToHost);
    cudaMemcpy(l.data(), lo, l.size() * 2, cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return printf("%s\n", cudaGetErrorString(e)), 1;
    double off = 0.0, norm = 0.0;
    std::vector<double> p(len), o(HD);
    for (int s = 0; s < ns; ++s)
        for (int head = 0; head < heads; ++head) {
            auto row = [&](int t, int v) { return &exact[(size_t)table[(size_t)s * pps + t / pt] * page + ((size_t)(v * kv + head / gqa) * pt + t % pt) * HD]; };
            const size_t at0 = ((size_t)s * heads + head) * HD;
            double top = -1e300, sum = 0.0;
            for (int t = 0; t < len; ++t) {
                double d = 0.0;
                for (int i = 0; i < HD; ++i) d += (double)q[at0 + i] * row(t, 0)[i];
                p[t] = d / std::sqrt((double)HD);
                top = std::max(top, p[t]);
            }
            std::fill(o.begin(), o.end(), 0.0);
            for (int t = 0; t < len; ++t) {
                const double w = std::exp(p[t] - top);
                sum += w;
                for (int i = 0; i < HD; ++i) o[i] += w * row(t, 1)[i];
            }
            for (int i = 0; i < HD; ++i) {
                const double d = (double)__half2float(h[at0 + i]) + (double)__half2float(l[at0 + i]) - o[i] / sum;
                off += d * d;
                norm += o[i] / sum * (o[i] / sum);
            }
        }
    printf("%.6g %d %d %d %d\n", std::sqrt(off / norm), cut.rounds, cut.spans, cut.shared, cut.own);
    return 0;
}

int main(int argc, char** argv) {
    if (argc != 10) return 2;
    const bool bf16 = !strcmp(argv[1], "bf16");
    int a[8];
    for (int i = 0; i < 8; ++i) a[i] = atoi(argv[2 + i]);
    if (a[0] == 128) return bf16 ? check<__nv_bfloat16, 128>(a[1], a[2], a[3], a[4], a[5], a[6], a[7]) : check<__half, 128>(a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
    if (a[0] == 64) return bf16 ? check<__nv_bfloat16, 64>(a[1], a[2], a[3], a[4], a[5], a[6], a[7]) : check<__half, 64>(a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
    return 2;
}
