// Host build of fft_core.cuh's two-stage transforms: both orders of the radices, run serially with the
// exchange matrix between the stages, for comparison with numpy.
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

extern "C" int fft_two(int n, int swapped, int inverse, const float* in, float* out) {
    const float2* i = reinterpret_cast<const float2*>(in);
    float2* o = reinterpret_cast<float2*>(out);
    switch (n) {
    case 192: return fft_n<192>(swapped, inverse, i, o);
    case 384: return fft_n<384>(swapped, inverse, i, o);
    }
    return -1;
}
