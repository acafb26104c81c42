// Host build of fft_core.cuh's two-stage transforms (both orders of the radices, run serially with the
// exchange matrix between the stages) and of the device passes' plans with a merged middle stage of radix
// 6, 12 or 24, scalar and paired, for comparison with numpy.
#include <cmath>
#include <vector>
#include "../../auto_gb300/csrc/fft_core.cuh"

using namespace lfft;

template <int N, int R1, int R2, bool INV>
static void run(const float2* in, float2* out, const float2* stw) {
    std::vector<float2> x(two_exchange(N));
    float2 v[32];
    for (int j = 0; j < N / R1; j++) {
        for (int m = 0; m < R1; m++) v[m] = in[j + m * (N / R1)];
        Dft<R1, INV>::run(v);
        two_store<R1>(x.data(), j, v);
    }
    for (int j = 0; j < N / R2; j++) {
        two_load<N, R2, INV>(x.data(), j, v, stw);
        for (int m = 0; m < R2; m++) out[j + m * (N / R2)] = v[m];
    }
}

template <int N>
static int fft_n(int swapped, int inverse, const float2* in, float2* out) {
    std::vector<float2> tw(TWN), stw(two_tw_size(N));
    for (int t = 0; t < TWN; t++) {
        const double a = -2.0 * M_PI * (double)t / (double)TWN;
        tw[t] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    fill_two_twiddles<N>(stw.data(), tw.data(), 0, 1);
    constexpr int A = two_stage(N).ra, B = two_stage(N).rb;
    static_assert(A * B == N, "two stages");
    if (swapped) inverse ? run<N, B, A, true>(in, out, stw.data()) : run<N, B, A, false>(in, out, stw.data());
    else inverse ? run<N, A, B, true>(in, out, stw.data()) : run<N, A, B, false>(in, out, stw.data());
    return 0;
}

template <int N, int I, bool INV, class T, class W>
static void run_plan(T* seq, const W* tw) {
    if constexpr (I < plan_len(N, ROW_PLAN)) {
        constexpr int R = plan_radix(N, I, ROW_PLAN), L = plan_L(N, I, ROW_PLAN);
        std::vector<T> v(N);
        for (int j = 0; j < N / R; j++) stage_load<N, R, L, INV>(seq, j, &v[j * R], tw + stage_tw_offset(N, I, ROW_PLAN));
        for (int j = 0; j < N / R; j++) stage_store<N, R, L>(seq, j, &v[j * R]);
        run_plan<N, I + 1, INV>(seq, tw);
    }
}

// paired: the input and its conjugate side by side
template <int N, bool INV>
static int plan_n(int paired, const float2* in, float2* out, const float2* tw) {
    if (paired) {
        std::vector<cpair> seq(seq_stride(N));
        std::vector<tw2> stw(tw_table_size(N, ROW_PLAN) + 1);
        fill_stage_twiddles<N, tw2, 0, ROW_PLAN>(stw.data(), tw, 0, 1);
        for (int i = 0; i < N; i++)
            seq[pad(i)] = cpair{make_float2(in[i].x, in[i].x), make_float2(-in[i].y, in[i].y)};
        run_plan<N, 0, INV>(seq.data(), stw.data());
        for (int i = 0; i < N; i++) out[i] = make_float2(seq[pad(i)].re.y, seq[pad(i)].im.y);
        return 0;
    }
    std::vector<float2> seq(seq_stride(N)), stw(tw_table_size(N, ROW_PLAN) + 1);
    fill_stage_twiddles<N, float2, 0, ROW_PLAN>(stw.data(), tw, 0, 1);
    for (int i = 0; i < N; i++) seq[pad(i)] = in[i];
    run_plan<N, 0, INV>(seq.data(), stw.data());
    for (int i = 0; i < N; i++) out[i] = seq[pad(i)];
    return 0;
}

extern "C" int fft_merged(int n, int paired, int inverse, const float* in, float* out) {
    const float2* i = reinterpret_cast<const float2*>(in);
    float2* o = reinterpret_cast<float2*>(out);
    std::vector<float2> tw(TWN);
    for (int t = 0; t < TWN; t++) {
        const double a = -2.0 * M_PI * (double)t / (double)TWN;
        tw[t] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    switch (n) {
#define CASE(N) case N: return inverse ? plan_n<N, true>(paired, i, o, tw.data()) : plan_n<N, false>(paired, i, o, tw.data());
        CASE(96) CASE(384) CASE(1536) CASE(3072) CASE(6144)
#undef CASE
    }
    return -1;
}

extern "C" int merged_plan(int n, int* out) {
    const Plan p = make_plan(n, ROW_PLAN);
    for (int i = 0; i < p.len; i++) out[i] = p.r[i];
    return p.len;
}

extern "C" int fft_two(int n, int swapped, int inverse, const float* in, float* out) {
    const float2* i = reinterpret_cast<const float2*>(in);
    float2* o = reinterpret_cast<float2*>(out);
    switch (n) {
    case 192: return fft_n<192>(swapped, inverse, i, o);
    case 384: return fft_n<384>(swapped, inverse, i, o);
    }
    return -1;
}
