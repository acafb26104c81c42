// Fused FP32 Lenia step on the CUDA cores: two launches per step.
//
// The reference's step is 4*log2(n)+5 full-grid dispatches (spectral.rs:199-264): load, log2 W
// x-stages, log2 H y-stages, spectrum copy, and per kernel multiply, inverse y, inverse x,
// convolved, then update.  Here the same mathematics is regrouped so that each grid sweep
// does as much as it can in shared memory:
//
//   column pass (per world, channel, tile of TC = 2 spectrum columns, kernel k reading it):
//       forward FFT along y  ->  x khat_k (real, even; includes 1/(W*H))  ->  inverse FFT along y
//   row pass (per world, block of 2 to 8 rows; Lenia: and target channel):
//       inverse real FFT along x of U_k  ->  growth, dt, clamp (spectral.rs:337-345)  ->
//       write state  ->  forward real FFT along x of the new rows  ->  write spectrum
//
// so one step reads and writes the half-spectrum twice and the state once.  Two real rows
// share one complex FFT (z = a + i b), and the real DC and Nyquist columns share spectrum
// column 0, so the half-spectrum takes exactly W*H*4 bytes per channel.
//
// The column pass is built twice: scalar (col_pass: a thread runs a butterfly of one column) and
// paired (col_pass_pair: a thread runs the same butterfly of both columns of the tile as f32x2
// pairs, half the threads and instructions); launch variant 2 selects the paired build, the default from
// 3072 to 6144.
#pragma once
#include <cuda_runtime.h>

#include "cache_hints.cuh"
#include "engine.cuh"
#include "fft_core.cuh"
#include "tc_ptx.cuh"

namespace lenia {
using namespace lfft;

// Programmatic dependent launch (LaunchOn::overlap): grid_wait returns when the kernel before this one has
// finished and its writes are visible (at once in a launch without overlap); grid_trigger
// (LaunchOn::early) lets the next kernel's CTAs start once every CTA of this one has called it or
// ended.  Every CTA of an overlapped pass waits, so a pass that has finished implies that every pass
// before it has.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// 16-byte asynchronous global -> shared copy: nothing is held in registers while it is in flight.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// f(Int<I>()) for I = 0..N-1, so that I (decltype(i)::value) can be a template argument.
template <int I>
struct Int {
    static constexpr int value = I;
    __host__ __device__ constexpr operator int() const { return I; }
};
template <int I, int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
    if constexpr (I < N) {
        f(Int<I>());
        static_for<I + 1, N>(f);
    }
}

// Stages [I, I1) of the transform of S sequences of length N in shared memory (stride
// seq_stride(N)), in place, by NT threads; stw holds the per-stage twiddle tables
// (fill_stage_twiddles).  Starts after the caller's barrier; ends with a barrier.
// MR: the plans (ROW_PLAN, COL_PLAN, or make_plan's radix cap): COL_PLAN in the scalar column pass only.
template <int N, int S, int NT, bool INV, int I, int I1, int MR = ROW_PLAN, class T, class W>
__device__ __forceinline__ void fft_stages(T* buf, const W* stw) {
    static_assert(MR != COL_PLAN || sizeof(T) == sizeof(float2), "radix-32 plans are built for scalar elements only");
    if constexpr (I < I1) {
        constexpr int R = plan_radix(N, I, MR);
        constexpr int L = plan_L(N, I, MR);
        constexpr int NB = N / R;
        constexpr int TOT = NB * S;
        constexpr int PER = (TOT + NT - 1) / NT;
        constexpr int SEQ = seq_stride(N);
        T v[PER][R];
#pragma unroll
        for (int p = 0; p < PER; p++) {
            const int b = threadIdx.x + p * NT;
            if ((TOT % NT) == 0 || b < TOT) {
                const int s = b / NB, j = b - s * NB;
                stage_load<N, R, L, INV>(buf + s * SEQ, j, v[p], stw + stage_tw_offset(N, I, MR));
            }
        }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < PER; p++) {
            const int b = threadIdx.x + p * NT;
            if ((TOT % NT) == 0 || b < TOT) {
                const int s = b / NB, j = b - s * NB;
                stage_store<N, R, L>(buf + s * SEQ, j, v[p]);
            }
        }
        __syncthreads();
        fft_stages<N, S, NT, INV, I + 1, I1, MR>(buf, stw);
    }
}

// ------------------------------------------------------------------ chained transforms
// Two transforms back to back (A, then B) with work on the values in between.  The last stage of A and
// the first of B share a radix R: A's leaves butterfly j holding the elements j + m*N/R (m < R) in
// natural order -- exactly the inputs of butterfly j of B's first stage.  So the work runs on those
// registers and B's first stage follows without a round trip through shared memory: two barriers and one
// shared-memory read/write sweep fewer than A, mid-pass, B.
// Scalar transforms of the sides fft_core.cuh's two_stage lists run A as RA, RB and B as RB, RA; the others run a
// plan whose first and last radix are equal, both ways.  The pieces, for either kind (sequences in
// shared memory in padded natural order before A and after B, stride seq_stride(N)):
//   chain_radix   R
//   fft_head      A's stages before its last one; ends with a barrier
//   chain_load    butterfly j of A's last stage
//   chain_store   the results of butterfly j of B's first stage (after a barrier, and before one)
//   fft_tail      B's other stages; ends with a barrier
template <int N, int MR = ROW_PLAN>
FFT_CHD constexpr bool fusable() {
    return is_two_stage(N, MR) || (plan_len(N, MR) >= 2 && plan_radix(N, 0, MR) == plan_radix(N, plan_len(N, MR) - 1, MR));
}
template <int N, int MR = ROW_PLAN>
FFT_CHD constexpr int chain_radix() { return is_two_stage(N, MR) ? two_stage(N, MR).rb : plan_radix(N, 0, MR); }
// Twiddle tables of a scalar transform: two-stage or per stage of the plan.
template <int N, int MR = ROW_PLAN>
FFT_CHD constexpr int tables_size() { return is_two_stage(N, MR) ? two_tw_size(N) : tw_table_size(N, MR); }
template <int N, int MR = ROW_PLAN>
__device__ __forceinline__ void fill_tables(float2* stw, const float2* tw, int nth) {
    if constexpr (is_two_stage(N, MR)) fill_two_twiddles<N>(stw, tw, threadIdx.x, nth);
    else fill_stage_twiddles<N, float2, 0, MR>(stw, tw, threadIdx.x, nth);
}

// One stage of S two-stage sequences, of radix R: the first of a transform (natural order in, exchange matrix out) or its
// second (exchange matrix in, natural order out).
template <int N, int R, int S, int NT, bool INV, bool SECOND>
__device__ __forceinline__ void two_stage_pass(float2* buf, const float2* stw) {
    constexpr int NB = N / R, TOT = NB * S, PER = (TOT + NT - 1) / NT, SEQ = seq_stride(N);
    static_assert(two_exchange(N) <= SEQ, "the exchange matrix takes the sequence's place");
    float2 v[PER][R];
#pragma unroll
    for (int p = 0; p < PER; p++) {
        const int b = threadIdx.x + p * NT;
        if ((TOT % NT) == 0 || b < TOT) {
            const int s = b / NB, j = b - s * NB;
            if constexpr (SECOND) two_load<N, R, INV>(buf + s * SEQ, j, v[p], stw);
            else stage_load<N, R, 1, INV>(buf + s * SEQ, j, v[p], stw);
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; p++) {
        const int b = threadIdx.x + p * NT;
        if ((TOT % NT) == 0 || b < TOT) {
            const int s = b / NB, j = b - s * NB;
            if constexpr (SECOND) stage_store<N, R, NB>(buf + s * SEQ, j, v[p]);
            else two_store<R>(buf + s * SEQ, j, v[p]);
        }
    }
    __syncthreads();
}

// Whole transforms in place.  SWAP: the order of B (RB, RA).
template <int N, int S, int NT, bool INV, bool SWAP, int MR = ROW_PLAN, class T, class W>
__device__ __forceinline__ void fft_seqs(T* buf, const W* stw) {
    if constexpr (is_two_stage(N, MR) && sizeof(T) == sizeof(float2)) {
        constexpr int R1 = SWAP ? two_stage(N, MR).rb : two_stage(N, MR).ra, R2 = N / R1;
        two_stage_pass<N, R1, S, NT, INV, false>(buf, stw);
        two_stage_pass<N, R2, S, NT, INV, true>(buf, stw);
    } else {
        fft_stages<N, S, NT, INV, 0, plan_len(N, MR), MR>(buf, stw);
    }
}

template <int N, int S, int NT, bool INV, int MR = ROW_PLAN>
__device__ __forceinline__ void fft_head(float2* buf, const float2* stw) {
    if constexpr (is_two_stage(N, MR)) two_stage_pass<N, two_stage(N, MR).ra, S, NT, INV, false>(buf, stw);
    else fft_stages<N, S, NT, INV, 0, plan_len(N, MR) - 1, MR>(buf, stw);
}
template <int N, bool INV, int MR = ROW_PLAN>
__device__ __forceinline__ void chain_load(const float2* seq, int j, float2* v, const float2* stw) {
    constexpr int LAST = plan_len(N, MR) - 1, R = chain_radix<N, MR>();
    if constexpr (is_two_stage(N, MR)) two_load<N, R, INV>(seq, j, v, stw);
    else stage_load<N, R, N / R, INV>(seq, j, v, stw + stage_tw_offset(N, LAST, MR));
}
template <int N, int MR = ROW_PLAN>
__device__ __forceinline__ void chain_store(float2* seq, int j, const float2* v) {
    constexpr int R = chain_radix<N, MR>();
    if constexpr (is_two_stage(N, MR)) two_store<R>(seq, j, v);
    else stage_store<N, R, 1>(seq, j, v);
}
template <int N, int S, int NT, bool INV, int MR = ROW_PLAN>
__device__ __forceinline__ void fft_tail(float2* buf, const float2* stw) {
    if constexpr (is_two_stage(N, MR)) two_stage_pass<N, two_stage(N, MR).ra, S, NT, INV, true>(buf, stw);
    else fft_stages<N, S, NT, INV, 1, plan_len(N, MR), MR>(buf, stw);
}

struct NoPre {
    __device__ void operator()(int, int) const {}
};

// A, mid(s, j, v) on the registers between (sequence s, elements j + m*N/R), B.  `pre(s, j)` runs just before
// the last stage of A.
template <int N, int S, int NT, bool INV_A, bool INV_B, int MR = ROW_PLAN, class Mid, class Pre = NoPre>
__device__ __forceinline__ void fft_fused(float2* buf, const float2* stw, Mid mid, Pre pre = Pre()) {
    static_assert(fusable<N, MR>(), "fusable plans only");
    constexpr int R = chain_radix<N, MR>(), NB = N / R;
    constexpr int TOT = NB * S, PER = (TOT + NT - 1) / NT, SEQ = seq_stride(N);
    fft_head<N, S, NT, INV_A, MR>(buf, stw);
    float2 v[PER][R];
#pragma unroll
    for (int p = 0; p < PER; p++) {
        const int b = threadIdx.x + p * NT;
        if ((TOT % NT) == 0 || b < TOT) {
            const int s = b / NB, j = b - s * NB;
            pre(s, j);  // global loads that mid needs, issued before the last stage of A
            chain_load<N, INV_A, MR>(buf + s * SEQ, j, v[p], stw);
            mid(s, j, v[p]);
            Dft<R, INV_B>::run(v[p]);  // B's first stage: L = 1, no twiddle
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; p++) {
        const int b = threadIdx.x + p * NT;
        if ((TOT % NT) == 0 || b < TOT) chain_store<N, MR>(buf + (b / NB) * SEQ, b % NB, v[p]);
    }
    __syncthreads();
    fft_tail<N, S, NT, INV_B, MR>(buf, stw);
}

// Shared memory of a pass: the sequences, then (float2-aligned) the twiddle tables.
template <int N, int MR = ROW_PLAN>
constexpr size_t stage_table_bytes() { return (size_t)(tables_size<N, MR>() + 1) * sizeof(float2); }

// The scalar column pass's plans: radix 32 where that saves a stage (1024 = 32.32 against 16.4.16: one
// shared-memory round trip fewer per transform; 8192 = 32.8.32), two stages at 192, 384 and 768, the merged plans at 96 and
// from 1536 up where the side has a 3 (3072 = 16.12.16), radix 16 elsewhere.  The column item holds its up to 32
// elements a thread in registers between stages; the row pass, which also holds the state values of its rows there, keeps
// radix 16 in its chained stages.
constexpr int CMR = COL_PLAN;

// Column pass, fused form: after the stage tables (16-byte aligned), the tile's TC khat columns.
template <int H>
FFT_CHD constexpr int khat_cols_stride() { return (H / 2 + 1 + 3) / 4 * 4; }
template <int H>
constexpr size_t col_khat_bytes() { return (size_t)TC * khat_cols_stride<H>() * sizeof(float); }
template <int H, int MR = CMR>
__device__ __forceinline__ float* col_khat_smem(float2* stw) {
    constexpr int TWS = tables_size<H, MR>();
    return reinterpret_cast<float*>(((uintptr_t)(stw + TWS) + 15) & ~(uintptr_t)15);
}

__device__ __forceinline__ float clamp01(float v) { return fminf(fmaxf(v, 0.0f), 1.0f); }

// Gaussian growth mapped to [-1, 1] (spectral.rs:341-344): 2 exp(-d^2/2) - 1, d = (u - mu)/sigma.
// Evaluated as 2 * 2^(-e^2) - 1 with e = u*k - mu*k, k = sqrt(log2(e)/2)/sigma: one FMA, one
// multiply, the hardware base-2 exponential (ex2.approx.ftz: a value below 2^-126 flushes to 0,
// which changes nothing because 2*2^(-e^2) - 1 then rounds to -1 either way) and one FMA.  Within
// 4e-7 of the direct form at the reference's parameters.
struct Growth {
    float k, mk;
    __device__ __forceinline__ Growth(float mu, float sigma) {
        k = 0.84932180028801904f / sigma;
        mk = mu * k;
    }
    __device__ __forceinline__ float operator()(float u) const {
        const float e = fmaf(u, k, -mk);
        float p;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p) : "f"(-e * e));
        return fmaf(2.0f, p, -1.0f);
    }
};

// 1 / (1 + e^(x k)) for a compile-time k, with the hardware base-2 exponential and reciprocal (one
// multiply, ex2, add, rcp).  A large x overflows e^(x k) to +inf, whose reciprocal is the 0 the
// logistic tends to; a value below 2^-126 flushes to 0 and the result rounds to 1 either way.
__device__ __forceinline__ float logistic_neg(float x, float k_log2e) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * k_log2e));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return r;
}

// SmoothLife update (spectral.rs:396-407): three logistic steps of width 4/AM and 4/AN.
__device__ __forceinline__ float smoothlife_update(float s, float c0, float c1) {
    const float B1 = 0.278f, B2 = 0.365f, D1 = 0.267f, D2 = 0.445f, DT = 0.1f;
    const float KM = 39.257007915345945f, KN = 206.09929155556621f;  // (4 / AM) log2(e), (4 / AN) log2(e)
    const float m = logistic_neg(0.5f - c0, KM);
    const float lo = B1 * (1.0f - m) + D1 * m, hi = B2 * (1.0f - m) + D2 * m;
    const float target = logistic_neg(lo - c1, KN) * (1.0f - logistic_neg(hi - c1, KN));
    return clamp01(s + DT * (2.0f * target - 1.0f));
}

// MNCA update (spectral.rs:461-472).
__device__ __forceinline__ float mnca_update(float s, float c0, float c1) {
    float o = s;
    if (c0 >= 0.210f && c0 <= 0.220f) o = 1.0f;
    if (c0 >= 0.350f && c0 <= 0.500f) o = 0.0f;
    if (c0 >= 0.750f && c0 <= 0.850f) o = 0.0f;
    if (c0 >= 0.120f && c0 <= 0.150f) o = 0.0f;
    if (c1 >= 0.100f && c1 <= 0.280f) o = 0.0f;
    if (c1 >= 0.430f && c1 <= 0.550f) o = 1.0f;
    return o;
}

// ---------------------------------------------------------------------------- row pass
//
// One CTA per item of 2S rows (S packed sequences, row pairs).  The single-kernel step uses S = 4 up to
// 1024 wide: an item then reads and writes each tile's spectrum as 128 contiguous bytes (8 rows x 16
// B) instead of 64, and on the 384-world batched workload the row pass went from 189 to 166 us a
// generation for the 1024 x 1024 class (512: 41 -> 34 us), the step from 1.75e11 to 1.87e11 cell-updates/s.
// Rows of 1536 to 4096 take S = 2: measured at 4096 x 4096, S = 4 (1024 threads, one CTA per SM) was 10% slower
// (row pass 76 against 68 us) and S = 1 (256 threads, three or four CTAs per SM) 4% slower (107 against 103 us a
// generation) than S = 2 (512 threads, two CTAs per SM).  From 6144 up S = 2 leaves one CTA an SM and S = 1 wins (6144 x 6144
// 378 -> 333 us a generation, 8192 x 8192 569 -> 528, with one-column columns at 8192).  The general step keeps a plane of W x 2S floats besides
// the sequences; from W = 2048 up it uses S = 1 (at S = 2 a 4096-wide item needed 138 KB of shared
// memory, one CTA per SM; MNCA at 4096 x 4096 measured 7% faster at S = 1), up to 1024 wide S = 4 (the
// 3-channel 1024 x 1024 world: 5.97e10 -> 6.33e10 channel-cell updates/s from S = 2, and 5% slower at
// S = 1 than at S = 2), in between S = 2.
// Threads of a row item of S sequences of length N: one first-stage butterfly per thread; for sides
// 3 * 2^k at least one per four radix-3 butterflies as well.  768 = 16.3.16 with 192 threads for four
// sequences ran its radix-3 stage in six rounds, the last a third full, and needed 128 registers a
// thread; with 256 it fits 64, and the batched workload's 768 x 768 row pass went from 104 to 89 us a
// generation (the step from 1.87e11 to 1.93e11 cell-updates/s).
// Two-stage sides: one butterfly of either stage.
FFT_CHD constexpr int seq_threads(int N, int S) {
    if (is_two_stage(N)) return S * two_tw_len(N);
    return N % 3 == 0 && N < 6144 && S * N / 12 > S * N / plan_radix(N, 0) ? S * N / 12 : S * N / plan_radix(N, 0);
}
FFT_CHD constexpr int row_seqs(int W, bool gen) { return gen ? (W >= 2048 ? 1 : (W <= 1024 ? 4 : 2)) : (W <= 1024 ? 4 : W >= 6144 ? 1 : 2); }
// Sequences a CTA holds: an item's, or from 768 up in variant 1 of the single-kernel step, which runs where the items
// leave SMs idle, half of them (two CTAs an item): one 4096 x 256 world 13.3 -> 10.0 us a generation, 1536 x 768 12.9 ->
// 11.8, 1024 x 256 8.2 -> 7.1, 768 x 768 9.4 -> 9.1, but 384 x 384 6.8 -> 9.8 and 256 x 256 5.5 -> 6.0.
FFT_CHD constexpr int row_cta_seqs(int W, int V, bool gen) {
    return V == 1 && !gen && W >= 768 && row_seqs(W, gen) > 1 ? row_seqs(W, gen) / 2 : row_seqs(W, gen);
}
template <int W, bool GEN, int V = 0>
constexpr int row_nt() {
    constexpr int n = seq_threads(W, row_cta_seqs(W, V, GEN));
    return n < 32 ? 32 : (n > 1024 ? 1024 : n);
}
// variant 0: at most 64 registers a thread (1024 threads an SM), 80 at 192 and 512 (which spill 40 bytes at 64: 63 worlds of
// 192 x 192 14.0 -> 13.5 us a generation, 41 of 512 x 512 55.5 -> 42.7, one 11.2 -> 6.6) and in the general step (which
// spilled at 64 at most sizes; three 256-thread CTAs an SM: three channels of 1024 x 1024 with nine kernels 43.4 -> 41.8);
// variant 1: at most 128
template <int W, int V, bool GEN>
constexpr int row_minb() {
    constexpr int t = V == 0 ? (GEN || W == 192 || W == 512 ? 768 : 1024) : 512, b = t / row_nt<W, GEN, V>();
    return b < 1 ? 1 : b > 32 ? 32 : b;
}
// 256-bit spectrum accesses, but 128-bit ones in the builds for a few rows of small worlds, whose launches wait for
// a single access's latency: one 256 x 256 world 5.9 -> 5.5 us a generation, 384 x 384 7.1 -> 6.8; against them
// 1024 worlds of 256 x 256 233 -> 222, one of 1024 x 1024 11.1 -> 10.3, 4096 x 4096 109.7 -> 103.0.
template <int W, int V>
constexpr bool row_wide() { return !(V == 1 && W <= 384); }
// Half-spectra of rows r0..r0+2S-1 (tile layout) <-> S packed complex sequences Z_p = A + iB with A = row
// r0+2p, B = row r0+2p+1, using Hermitian symmetry for k > W/2.
// A lane moves 32 bytes: both columns (kx = 2t, 2t+1) of one tile t for one row pair p, consecutive lanes on the
// pairs of a tile.  A half-warp's shared-memory accesses have stride 2 within a pair; with the sequences 1 mod 16
// apart, and at S = 4 the even tiles in one half-warp and the odd in the other, they touch all banks once (at S = 1
// every other eight lanes take their second column first instead).  The row pass is bound by L1 wavefronts
// (67-77% of their peak at 4096 and 8192), and as 8-byte accesses -- a lane per column and row -- the spectrum
// took twice the wavefronts and four times the instructions.
template <int W, int S, int NT>
struct RowLanes {
    static constexpr int TILES = W / 4, G = S == 4 ? 8 : 1;  // tiles are dealt in groups of G
    static constexpr int E = (TILES + G - 1) / G * G * S, IT = (E + NT - 1) / NT;
    // kx moves by D an iteration; a multiple of 16 moves padded positions by D + D / 16
    static constexpr int D = 2 * NT / S, O = D + D / 16;
    static constexpr bool STEP = NT % (G * S) == 0 && D % 16 == 0;
    static constexpr bool FULL = TILES % G == 0 && IT * NT == E;
};
template <int S>
__device__ __forceinline__ int row_tile(int e) {
    return S == 4 ? (e >> 5) * 8 + 2 * ((e >> 2) & 3) + ((e >> 4) & 1) : e / S;
}

template <int W, int S, int NT, bool CG, bool WIDE>
__device__ __forceinline__ void load_rows_spectrum(float2* Z, const float2* __restrict__ sp, int H, int r0) {
    using L = RowLanes<W, S, NT>;
    constexpr int SEQ = seq_stride(W);
    float2 v[L::IT][4];
#pragma unroll
    for (int i = 0; i < L::IT; i++) {
        const int e = threadIdx.x + i * NT, t = row_tile<S>(e), p = e % S;
        if (L::FULL || t < L::TILES)
            hint::ld8c<CG, WIDE>(v[i], sp + ((size_t)t * H + r0 + 2 * p) * TC);
    }
    const int t0 = row_tile<S>(threadIdx.x), p0 = threadIdx.x % S;
    float2* za0 = Z + p0 * SEQ + pad(2 * t0);
    float2* zb0 = Z + p0 * SEQ + pad(W - 2 * t0);
    float2* zc0 = Z + p0 * SEQ + pad(W - 2 * t0 - 1);
#pragma unroll
    for (int i = 0; i < L::IT; i++) {
        const int e = threadIdx.x + i * NT, t = row_tile<S>(e), p = e % S;
        const bool swap = S == 1 && (threadIdx.x & 8);
        if (!L::FULL && t >= L::TILES) continue;
        float2* z = Z + p * SEQ;
        // kx = 2t at za and (mirrored) zb, kx = 2t + 1 at za + 1 and zc
        float2* za = L::STEP ? za0 + i * L::O : z + pad(2 * t);
        float2* zb = L::STEP ? zb0 - i * L::O : z + pad(W - 2 * t);
        float2* zc = L::STEP ? zc0 - i * L::O : z + pad(W - 2 * t - 1);
        const float2 A0 = v[i][0], A1 = v[i][1], B0 = v[i][2], B1 = v[i][3];
        const float2 p0_ = make_float2(A0.x - B0.y, A0.y + B0.x), m0 = make_float2(A0.x + B0.y, B0.x - A0.y);
        const float2 p1 = make_float2(A1.x - B1.y, A1.y + B1.x), m1 = make_float2(A1.x + B1.y, B1.x - A1.y);
        if (t == 0) {  // column 0 packs DC and Nyquist
            z[pad(0)] = make_float2(A0.x, B0.x);
            z[pad(W / 2)] = make_float2(A0.y, B0.y);
            za[1] = p1;
            *zc = m1;
        } else {
            za[swap ? 1 : 0] = swap ? p1 : p0_;
            za[swap ? 0 : 1] = swap ? p0_ : p1;
            *(swap ? zc : zb) = swap ? m1 : m0;
            *(swap ? zb : zc) = swap ? m0 : m1;
        }
    }
}

// S packed complex spectra Z_p = FFT(a + ib) -> half-spectra of rows r0+2p (A) and r0+2p+1 (B).
template <int W, int S, int NT, bool WIDE>
__device__ __forceinline__ void store_rows_spectrum(const float2* Z, float2* __restrict__ sp, int H, int r0) {
    using L = RowLanes<W, S, NT>;
    constexpr int SEQ = seq_stride(W);
    const int t0 = row_tile<S>(threadIdx.x), p0 = threadIdx.x % S;
    const float2* za0 = Z + p0 * SEQ + pad(2 * t0);
    const float2* zb0 = Z + p0 * SEQ + pad(W - 2 * t0);
    const float2* zc0 = Z + p0 * SEQ + pad(W - 2 * t0 - 1);
#pragma unroll
    for (int i = 0; i < L::IT; i++) {
        const int e = threadIdx.x + i * NT, t = row_tile<S>(e), p = e % S;
        const bool swap = S == 1 && (threadIdx.x & 8);
        if (!L::FULL && t >= L::TILES) continue;
        const float2* z = Z + p * SEQ;
        const float2* za = L::STEP ? za0 + i * L::O : z + pad(2 * t);
        const float2* zb = L::STEP ? zb0 - i * L::O : z + pad(W - 2 * t);
        const float2* zc = L::STEP ? zc0 - i * L::O : z + pad(W - 2 * t - 1);
        const float2* zm = t == 0 ? za : zb;  // column 0 has no mirror
        const float2 f = za[swap ? 1 : 0], s = za[swap ? 0 : 1], g = *(swap ? zc : zm), h = *(swap ? zm : zc);
        const float2 a0 = swap ? s : f, a1 = swap ? f : s, b0 = swap ? h : g, b1 = swap ? g : h;
        float2 A, B;
        if (t == 0) {
            const float2 zn = z[pad(W / 2)];
            A = make_float2(a0.x, zn.x);
            B = make_float2(a0.y, zn.y);
        } else {
            A = make_float2(0.5f * (a0.x + b0.x), 0.5f * (a0.y - b0.y));
            B = make_float2(0.5f * (a0.y + b0.y), -0.5f * (a0.x - b0.x));
        }
        hint::st8<WIDE>(sp + ((size_t)t * H + r0 + 2 * p) * TC, A, make_float2(0.5f * (a1.x + b1.x), 0.5f * (a1.y - b1.y)), B,
                  make_float2(0.5f * (a1.y + b1.y), -0.5f * (a1.x - b1.x)));
    }
}

// Row-pass modes that run outside the step (after state writes, and for U-field reads).  Not
// inlined, so that their registers do not add to the step path's.
template <int W, int NT, int S>
__device__ __noinline__ void row_item_forward(float2* Z, const float2* stw, const DevWorld& wd, int r0, int d0, int d1) {
    constexpr int SEQ = seq_stride(W);
    const int H = wd.H;
    const size_t plane = (size_t)W * H, cplane = (size_t)(W / 2) * H;
    for (int d = d0; d < d1; d++) {
        const float* st = wd.state + d * plane + (size_t)r0 * W;
        constexpr int IT = (S * W + NT - 1) / NT;
        float a[IT], b[IT];
#pragma unroll
        for (int i = 0; i < IT; i++) {
            const int e = threadIdx.x + i * NT, p = e / W, x = e - p * W;
            if (IT * NT == S * W || e < S * W) {
                a[i] = st[(2 * p) * W + x];
                b[i] = st[(2 * p + 1) * W + x];
            }
        }
#pragma unroll
        for (int i = 0; i < IT; i++) {
            const int e = threadIdx.x + i * NT, p = e / W, x = e - p * W;
            if (IT * NT == S * W || e < S * W) Z[p * SEQ + pad(x)] = make_float2(a[i], b[i]);
        }
        __syncthreads();
        fft_seqs<W, S, NT, false, true>(Z, stw);
        store_rows_spectrum<W, S, NT, false>(Z, wd.spec + d * cplane, H, r0);
        __syncthreads();
    }
}

template <int W, int NT, int S>
__device__ __noinline__ void row_item_u(float2* Z, const float2* stw, const DevWorld& wd, int r0, int d0, bool per_chan) {
    constexpr int SEQ = seq_stride(W);
    const int H = wd.H, K = wd.K;
    const size_t plane = (size_t)W * H, cplane = (size_t)(W / 2) * H;
    for (int k = 0; k < K; k++) {
        if (per_chan && wd.kern[k].dst != d0) continue;
        load_rows_spectrum<W, S, NT, false, false>(Z, wd.conv + k * cplane, H, r0);
        __syncthreads();
        fft_seqs<W, S, NT, true, false>(Z, stw);
        float* u = wd.u_out + k * plane + (size_t)r0 * W;
        for (int e = threadIdx.x; e < S * W; e += NT) {
            const int p = e / W, x = e - p * W;
            const float2 z = Z[p * SEQ + pad(x)];
            u[(2 * p) * W + x] = z.x;
            u[(2 * p + 1) * W + x] = z.y;
        }
        __syncthreads();
    }
}

// The one-channel, one-kernel Lenia row step of rows r0..r0+2S-1 of world wd: inverse row FFT of U, growth,
// dt update and clamp against the state, forward row FFT of the new rows.  Z: the S packed
// sequences, stw: the stage tables.  CG: spectrum and state loads bypass L1 (the persistent step,
// where another CTA of the same launch wrote them).
template <int W, int NT, int S, bool CG, bool WIDE>
__device__ __forceinline__ void row_item_simple(const DevWorld& wd, int r0, float2* Z, const float2* stw, bool early = false) {
    constexpr int ROWS = 2 * S;
    const int H = wd.H;
    const DevKernel kp = wd.kern[0];
    const float dtw = wd.dt * kp.weight;
    const Growth growth(kp.mu, kp.sigma);
    float* st = wd.state + (size_t)r0 * W;
    const uint64_t stream = hint::policy_stream();
    // The growth update runs in registers between the inverse and the forward row FFT (every
    // built width has a plan with equal first and last radix).  The item's state rows are
    // pulled into L2 when the CTA starts, and each thread's 2 x R state values are loaded into
    // registers just before the last inverse stage.
    static_assert(fusable<W>(), "row widths need a plan with equal first and last radix");
    constexpr int R = chain_radix<W>(), NB = W / R;
    static_assert(S * NB <= NT, "one butterfly per thread in the fused stage");
    if (threadIdx.x == 0) tc::bulk_prefetch_l2(st, ROWS * W * (uint32_t)sizeof(float));
    if constexpr (!CG) grid_wait();
    load_rows_spectrum<W, S, NT, CG, WIDE>(Z, wd.conv, H, r0);
    __syncthreads();
    float sa[R], sb[R];
    fft_fused<W, S, NT, true, false>(
        Z, stw,
        [&](int s, int j, float2* v) {
            float* ga = st + (2 * s) * W + j;
            static_for<0, R>([&](auto m) {
                const float n0 = __saturatef(fmaf(dtw, growth(v[m].x), sa[m]));
                const float n1 = __saturatef(fmaf(dtw, growth(v[m].y), sb[m]));
                hint::st1_at<decltype(m)::value * NB * 4>(ga, n0, stream);
                hint::st1_at<(W + decltype(m)::value * NB) * 4>(ga, n1, stream);
                v[m] = make_float2(n0, n1);
            });
        },
        [&](int s, int j) {
            const float* ga = st + (2 * s) * W + j;
            static_for<0, R>([&](auto m) {
                sa[m] = hint::ld1_atc<decltype(m)::value * NB * 4, CG>(ga, stream);
                sb[m] = hint::ld1_atc<(W + decltype(m)::value * NB) * 4, CG>(ga, stream);
            });
        });
    if (!CG && early) grid_trigger();
    store_rows_spectrum<W, S, NT, WIDE>(Z, wd.spec, H, r0);
}

// GEN: the instantiation for size classes with worlds that need the general step (several
// channels or kernels, SmoothLife, MNCA).  Without it the kernel carries only the one-channel,
// one-kernel Lenia step (and the forward and U modes), so the general path's register pressure
// does not set the budget of the common path.
// WIDE: whether the spectrum moves in 256-bit accesses (row_wide; never in the noinline modes above, see hint::st8).
template <int W, int NT, int MINB, int S, bool GEN, bool WIDE>
__global__ void __launch_bounds__(NT, MINB) row_pass(const DevWorld* __restrict__ worlds, const RowItem* __restrict__ items,
                                                int mode, const float2* __restrict__ tw, bool early) {
    constexpr int ROWS = 2 * S, SPLIT = row_seqs(W, GEN) / S;  // CTAs an item
    extern __shared__ float4 smem_raw[];
    constexpr int SEQ = seq_stride(W);
    float2* Z = reinterpret_cast<float2*>(smem_raw);
    float2* stw = Z + (GEN ? 2 : 1) * S * SEQ;
    const RowItem it = items[blockIdx.x / SPLIT];
    const DevWorld& wd = worlds[it.world];
    fill_tables<W>(stw, tw, NT);
    const int H = wd.H, C = wd.C, K = wd.K, r0 = it.row0 + ROWS * (blockIdx.x % SPLIT);
    const size_t plane = (size_t)W * H, cplane = (size_t)(W / 2) * H;
    // Lenia items cover one target channel; SmoothLife and MNCA items every channel
    const bool per_chan = wd.rule == LENIA_RULE_LENIA;
    const int d0 = per_chan ? it.chan : 0, d1 = per_chan ? it.chan + 1 : C;

    if constexpr (GEN) grid_wait();
    if (mode == MODE_FORWARD) {
        row_item_forward<W, NT, S>(Z, stw, wd, r0, d0, d1);
        return;
    }
    if (mode == MODE_U) {
        row_item_u<W, NT, S>(Z, stw, wd, r0, d0, per_chan);
        return;
    }

    if constexpr (!GEN) {
        row_item_simple<W, NT, S, false, WIDE>(wd, r0, Z, stw, early);
        return;
    }

    // General: several channels and/or kernels, or SmoothLife / MNCA (one channel, two kernels); also
    // any one-kernel world that shares a size class with such worlds.
    // Every kernel of the item but the last leaves its result in one shared-memory plane, straight
    // from the registers of its last inverse stage: Lenia adds its weighted growth, SmoothLife and
    // MNCA keep the first kernel's U.  The last kernel runs chained (fft_fused): its last inverse
    // stage, the rule's update with the plane and the state, and the first forward stage stay in
    // registers.  A thread owns the same cells (sequence s, x = j + m*N/R) in all of these stages,
    // so the plane needs no barrier of its own.  It lies where the second kernel's sequences do below.
    const int rule = wd.rule;
    constexpr int R = chain_radix<W>(), NB = W / R;
    static_assert(fusable<W>(), "row widths need a plan with equal first and last radix");
    static_assert(S * NB <= NT, "one butterfly per thread in the chained stages");
    float* acc = reinterpret_cast<float*>(Z + S * SEQ);  // [ROWS][W]
    int nk = 0, klast = -1;
    for (int k = 0; k < K; k++)
        if (!per_chan || wd.kern[k].dst == d0) nk++, klast = k;
    float* st = wd.state + d0 * plane + (size_t)r0 * W;
    if (nk == 0) {
        // no kernel targets this channel: the update is the clamp alone
        for (int e = threadIdx.x; e < ROWS * W; e += NT) st[e] = clamp01(st[e]);
        __syncthreads();
        row_item_forward<W, NT, S>(Z, stw, wd, r0, d0, d0 + 1);
        return;
    }
    if (threadIdx.x == 0) tc::bulk_prefetch_l2(st, ROWS * W * (uint32_t)sizeof(float));
    const uint64_t stream = hint::policy_stream();
    // Two kernels up to 128 wide: the launch is bound by an item's latency, so both spectra are loaded at once, both inverse
    // transforms share their barriers (2S sequences), and nothing goes through the plane.  Same bits.  SmoothLife 64 x 64
    // 6.3 -> 5.2 us a generation, 128 x 1024 9.3 -> 8.3, two channels of 128 x 128 6.6 -> 6.0.  Wider items hold 16 elements
    // a thread and lose: 256 x 256 10.0 -> 12.6, 512 x 512 11.5 -> 15.3, 2048 x 2048 48.5 -> 51.0.
    constexpr bool PAIR = W <= 128 && NT * MINB <= 512;
    if (PAIR && nk == 2) {
        int k0 = 0;
        while (per_chan && wd.kern[k0].dst != d0) k0++;
        const DevKernel kp = wd.kern[k0], kq = wd.kern[klast];
        load_rows_spectrum<W, S, NT, false, WIDE>(Z, wd.conv + k0 * cplane, H, r0);
        load_rows_spectrum<W, S, NT, false, WIDE>(Z + S * SEQ, wd.conv + klast * cplane, H, r0);
        __syncthreads();
        fft_head<W, 2 * S, NT, true>(Z, stw);
        const Growth gp(kp.mu, kp.sigma), gq(kq.mu, kq.sigma);
        const float dt = wd.dt;
        const int s = threadIdx.x / NB, j = threadIdx.x - s * NB;
        const bool on = S * NB == NT || (int)threadIdx.x < S * NB;
        float2 v[R];
        if (on) {
            float sa[R], sb[R];
            float* ga = st + (2 * s) * W + j;
#pragma unroll
            for (int m = 0; m < R; m++) {
                sa[m] = hint::ld1(ga + m * NB, stream);
                sb[m] = hint::ld1(ga + W + m * NB, stream);
            }
            float2 u[R];
            chain_load<W, true>(Z + s * SEQ, j, u, stw);
            chain_load<W, true>(Z + (S + s) * SEQ, j, v, stw);
#pragma unroll
            for (int m = 0; m < R; m++) {
                float n0, n1;
                if (rule == LENIA_RULE_LENIA) {
                    n0 = clamp01(sa[m] + dt * __fmaf_rn(kq.weight, gq(v[m].x), __fmul_rn(kp.weight, gp(u[m].x))));
                    n1 = clamp01(sb[m] + dt * __fmaf_rn(kq.weight, gq(v[m].y), __fmul_rn(kp.weight, gp(u[m].y))));
                } else if (rule == LENIA_RULE_SMOOTHLIFE) {
                    n0 = smoothlife_update(sa[m], u[m].x, v[m].x);
                    n1 = smoothlife_update(sb[m], u[m].y, v[m].y);
                } else {
                    n0 = mnca_update(sa[m], u[m].x, v[m].x);
                    n1 = mnca_update(sb[m], u[m].y, v[m].y);
                }
                hint::st1(ga + m * NB, n0, stream);
                hint::st1(ga + W + m * NB, n1, stream);
                v[m] = make_float2(n0, n1);
            }
            Dft<R, false>::run(v);
        }
        __syncthreads();
        if (on) chain_store<W>(Z + s * SEQ, j, v);
        __syncthreads();
        fft_tail<W, S, NT, false>(Z, stw);
        if (early) grid_trigger();
        store_rows_spectrum<W, S, NT, WIDE>(Z, wd.spec + d0 * cplane, H, r0);
        return;
    }
    bool first = true;
    for (int k = 0; k < klast; k++) {
        const DevKernel kp = wd.kern[k];
        if (per_chan && kp.dst != d0) continue;
        const Growth growth(kp.mu, kp.sigma);
        load_rows_spectrum<W, S, NT, false, WIDE>(Z, wd.conv + k * cplane, H, r0);
        __syncthreads();
        fft_head<W, S, NT, true>(Z, stw);
        if ((int)threadIdx.x < S * NB) {
            const int s = threadIdx.x / NB, j = threadIdx.x - s * NB;
            float2 v[R];
            chain_load<W, true>(Z + s * SEQ, j, v, stw);
            float* a = acc + (2 * s) * W + j;
#pragma unroll
            for (int m = 0; m < R; m++) {
                if (rule == LENIA_RULE_LENIA) {
                    const float g0 = __fmul_rn(kp.weight, growth(v[m].x)), g1 = __fmul_rn(kp.weight, growth(v[m].y));
                    a[m * NB] = first ? g0 : a[m * NB] + g0;
                    a[W + m * NB] = first ? g1 : a[W + m * NB] + g1;
                } else {
                    a[m * NB] = v[m].x;
                    a[W + m * NB] = v[m].y;
                }
            }
        }
        first = false;
        __syncthreads();  // Z is rewritten by the next kernel
    }
    const DevKernel kp = wd.kern[klast];
    const Growth growth(kp.mu, kp.sigma);
    const float dt = wd.dt;
    const bool have_acc = nk > 1;
    load_rows_spectrum<W, S, NT, false, WIDE>(Z, wd.conv + klast * cplane, H, r0);
    __syncthreads();
    float sa[R], sb[R];
    fft_fused<W, S, NT, true, false>(
        Z, stw,
        [&](int s, int j, float2* v) {
            float* ga = st + (2 * s) * W + j;
            const float* a = acc + (2 * s) * W + j;
#pragma unroll
            for (int m = 0; m < R; m++) {
                float n0, n1;
                if (rule == LENIA_RULE_LENIA) {
                    const float g0 = growth(v[m].x), g1 = growth(v[m].y);
                    const float t0 = have_acc ? __fmaf_rn(kp.weight, g0, a[m * NB]) : kp.weight * g0;
                    const float t1 = have_acc ? __fmaf_rn(kp.weight, g1, a[W + m * NB]) : kp.weight * g1;
                    n0 = clamp01(sa[m] + dt * t0);
                    n1 = clamp01(sb[m] + dt * t1);
                } else if (rule == LENIA_RULE_SMOOTHLIFE) {
                    n0 = smoothlife_update(sa[m], a[m * NB], v[m].x);
                    n1 = smoothlife_update(sb[m], a[W + m * NB], v[m].y);
                } else {
                    n0 = mnca_update(sa[m], a[m * NB], v[m].x);
                    n1 = mnca_update(sb[m], a[W + m * NB], v[m].y);
                }
                hint::st1(ga + m * NB, n0, stream);
                hint::st1(ga + W + m * NB, n1, stream);
                v[m] = make_float2(n0, n1);
            }
        },
        [&](int s, int j) {
            const float* ga = st + (2 * s) * W + j;
#pragma unroll
            for (int m = 0; m < R; m++) {
                sa[m] = hint::ld1(ga + m * NB, stream);
                sb[m] = hint::ld1(ga + W + m * NB, stream);
            }
        });
    if (early) grid_trigger();
    store_rows_spectrum<W, S, NT, WIDE>(Z, wd.spec + d0 * cplane, H, r0);
}

// ---------------------------------------------------------------------------- column pass

// Column 0 of tile 0 packs the DC column (real part) and the Nyquist column (imaginary part): both are
// real sequences, so with Z = FFT_y(packed), K0 and KN their kernel spectra,
// Z'[ky] = Z[ky] (K0 + KN)/2 + conj(Z[-ky]) (K0 - KN)/2.  One rounding order, whoever computes it.
__device__ __forceinline__ float2 packed_times_khat(float2 z, float2 zm, float K0, float KN) {
    const float a = 0.5f * (K0 + KN), b = 0.5f * (K0 - KN);
    return make_float2(__fmaf_rn(z.x, a, __fmul_rn(zm.x, b)), __fmaf_rn(z.y, a, -__fmul_rn(zm.y, b)));
}

// X (TC sequences of length H in padded natural order, the forward spectrum of tile 0) times khat, in place.
template <int H, int NT>
__device__ __forceinline__ void multiply_khat(float2* X, const float* __restrict__ kh, int HQ, int W) {
    constexpr int SEQ = seq_stride(H);
    for (int ky = threadIdx.x; ky < H; ky += NT) {
        float2& z = X[SEQ + pad(ky)];
        z = cscale(z, kh[HQ + (ky <= H / 2 ? ky : H - ky)]);
    }
    for (int ky = threadIdx.x; ky <= H / 2; ky += NT) {
        const float K0 = kh[ky], KN = kh[(size_t)(W / 2) * HQ + ky];
        const int km = (H - ky) % H;
        const float2 z = X[pad(ky)], zm = X[pad(km)];
        X[pad(ky)] = packed_times_khat(z, zm, K0, KN);
        if (km != ky) X[pad(km)] = packed_times_khat(zm, z, K0, KN);
    }
}

// Stride between a column item's two sequences in shared memory: 8 mod 16 float2, so that the eight
// butterflies of both columns that a half-warp works on (see col_chained) touch all 32 banks once.
FFT_CHD constexpr int col_values(int n) { return n + (is_two_stage(n, CMR) && two_tw_len(n) > n / 16 ? two_tw_len(n) : n / 16); }
FFT_CHD constexpr int col_stride(int n) { return col_values(n) + (24 - col_values(n) % 16) % 16; }

// Stages [I, I1) of both columns of a tile in shared memory, as fft_stages, but with the column in the
// lowest bit of the butterfly index.
template <int N, int NT, bool INV, int I, int I1, int MR, int NC>
__device__ __forceinline__ void col_stages(float2* X, const float2* stw) {
    if constexpr (I < I1) {
        constexpr int R = plan_radix(N, I, MR), L = plan_L(N, I, MR);
        constexpr int TOT = NC * (N / R), PER = (TOT + NT - 1) / NT, CS = col_stride(N);
        float2 v[PER][R];
#pragma unroll
        for (int p = 0; p < PER; p++) {
            const int b = threadIdx.x + p * NT;
            if ((TOT % NT) == 0 || b < TOT)
                stage_load<N, R, L, INV>(X + (b % NC) * CS, b / NC, v[p], stw + stage_tw_offset(N, I, MR));
        }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < PER; p++) {
            const int b = threadIdx.x + p * NT;
            if ((TOT % NT) == 0 || b < TOT) stage_store<N, R, L>(X + (b % NC) * CS, b / NC, v[p]);
        }
        __syncthreads();
        col_stages<N, NT, INV, I + 1, I1, MR, NC>(X, stw);
    }
}

// The chained column item.  The first stage of a plan reads elements j + m H/R and the last stage
// leaves butterfly j the same elements, so with thread t on butterfly j = t / 2 of column t % 2 a
// warp's access to the tile (H rows of two columns) is 256 contiguous bytes: the forward transform's
// first stage takes its inputs straight from global memory and the inverse's last stage writes its
// outputs there.  That leaves 2 (stages - 1) sweeps of the tile through shared memory and
// 4 stages - 5 barriers, two sweeps and four barriers fewer than staging the tile both ways.  The item is
// bound by shared-memory instructions and barriers; measured, per generation: 60 worlds of 384 x 384
// 60.7 -> 55.3 us, 41 of 512 x 512 47.2 -> 44.7, one of 4096 x 4096 107.5 -> 103.3, of 8192 x 8192 576 -> 552.
// Tile 0, whose column 0 packs two real columns, runs the same way with one exchange through shared memory in
// the middle (khn: the Nyquist column's kernel spectrum; null in every other tile).  As a separate item of whole
// transforms and tile sweeps it took about twice as long as the others and was the last to finish in every launch
// that fits the GPU: one 512 x 512 world 8.9 -> 7.1 us a generation, 1024 x 1024 13.8 -> 10.7, 2048 x 1024 20.2 -> 16.0.
template <int H, int NT, bool CG, int MR, int NC>
__device__ __forceinline__ void col_chained(float2* X, const float2* stw, const float2* __restrict__ src,
                                            float2* __restrict__ dst, const float* ksm, const float* __restrict__ khn,
                                            int c0, bool early) {
    constexpr bool TWO = is_two_stage(H, MR);
    // radix of the stages at the tile (first of the forward transform, last of the inverse) and in the middle
    constexpr int RT = TWO ? two_stage(H, MR).ra : plan_radix(H, 0, MR), RM = chain_radix<H, MR>();
    constexpr int NT0 = H / RT, NM = H / RM, LAST = plan_len(H, MR) - 1, CS = col_stride(H);
    constexpr int HQC = khat_cols_stride<H>();
    static_assert(TC == 2 && fusable<H, MR>() && NC * NT0 <= NT && NC * NM <= NT, "one outer butterfly per thread and column");
    const int c = c0 + threadIdx.x % NC, j = threadIdx.x / NC;
    const bool tile = NC * NT0 == NT || threadIdx.x < NC * NT0, mid = NC * NM == NT || threadIdx.x < NC * NM;
    float2* Xc = X + (threadIdx.x % NC) * CS;
    if (tile) {
        float2 v[RT];
        const uint64_t keep = hint::policy_keep();
#pragma unroll
        for (int m = 0; m < RT; m++) v[m] = hint::ld2c<CG>(src + TC * j + c + TC * NT0 * m, keep);
        Dft<RT, false>::run(v);
        if constexpr (TWO) two_store<RT>(Xc, j, v);
        else stage_store<H, RT, 1>(Xc, j, v);
    }
    cp_async_wait_all();  // the khat columns
    __syncthreads();
    if constexpr (!TWO) col_stages<H, NT, false, 1, LAST, MR, NC>(X, stw);
    float2 v[RM];
    if (mid) {
        chain_load<H, false, MR>(Xc, j, v, stw);
        const float* kc = ksm + (threadIdx.x % NC) * HQC;
        if (khn == nullptr || c == 1) {
#pragma unroll
            for (int m = 0; m < RM; m++) {
                const int ky = j + m * NM;
                v[m] = cscale(v[m], kc[ky <= H / 2 ? ky : H - ky]);
            }
        }
    }
    if (khn != nullptr) {
        // tile 0 (the same for the whole CTA): column 0's values meet their mirrors through shared memory
        __syncthreads();
        if (mid && c == 0)
#pragma unroll
            for (int m = 0; m < RM; m++) X[j + m * NM] = v[m];
        __syncthreads();
        if (mid && c == 0)
#pragma unroll
            for (int m = 0; m < RM; m++) {
                const int ky = j + m * NM, kk = ky <= H / 2 ? ky : H - ky;
                v[m] = packed_times_khat(v[m], X[(H - ky) % H], ksm[kk], khn[kk]);
            }
    }
    if (mid) Dft<RM, true>::run(v);
    __syncthreads();
    if (mid) chain_store<H, MR>(Xc, j, v);
    __syncthreads();
    if (!CG && early) grid_trigger();
    if constexpr (!TWO) col_stages<H, NT, true, 1, LAST, MR, NC>(X, stw);
    if (tile) {
        float2 u[RT];
        if constexpr (TWO) two_load<H, RT, true>(Xc, j, u, stw);
        else stage_load<H, RT, NT0, true>(Xc, j, u, stw + stage_tw_offset(H, LAST, MR));
        const uint64_t keep = hint::policy_keep();
#pragma unroll
        for (int m = 0; m < RT; m++) hint::st2(dst + TC * j + c + TC * NT0 * m, u[m], keep);
    }
}

// A tile's two khat columns (rows of HQ floats) into shared memory, khat_cols_stride apart: asynchronous
// 16-byte copies where the rows allow it (khat_stride rows; the caller waits), else plain loads (lenia_step_noalloc's
// callers pass rows of H/2 + 1).
template <int H, int NT, int NC = TC>
__device__ __forceinline__ void copy_khat(float* ksm, const float* __restrict__ kh, int HQ) {
    constexpr int HQC = khat_cols_stride<H>();
    if (HQ == HQC && ((uintptr_t)kh & 15) == 0) {
        for (int e = threadIdx.x; e < NC * HQC / 4; e += NT) cp_async16(ksm + 4 * e, kh + 4 * e);
    } else {
        for (int e = threadIdx.x; e < NC * (H / 2 + 1); e += NT) {
            const int c = e / (H / 2 + 1), y = e - c * (H / 2 + 1);
            ksm[c * HQC + y] = kh[(size_t)c * HQ + y];
        }
    }
}

// One column item: tile `tile` (TC spectrum columns) of channel `chan`, convolved with kernel
// `kernel` (which reads that channel).  A channel read by several kernels has one item per kernel, each
// repeating the channel's forward column transform: that keeps every item on the chained path and
// multiplies the items, which the multichannel world needs more than it needs the saved transforms.
// CG: the tile loads bypass L1 (the persistent step, where another CTA of the same launch wrote them).
// NC: the columns of the tile this CTA takes, from c0 on.
template <int H, int NT, bool CG, int MR = CMR, int NC = TC>
__device__ __forceinline__ void col_item(const DevWorld& wd, const ColItem it, float2* X, float2* stw, int c0 = 0,
                                         bool early = false) {
    const int W = wd.W, c = it.chan, t = it.tile, k = it.kernel, HQ = wd.HQ;
    const size_t cplane = (size_t)(W / 2) * H;
    const float2* src = wd.spec + c * cplane + (size_t)t * H * TC;
    // The khat multiply runs in registers between the forward and the inverse column FFT; the tile's two
    // khat columns (HQ floats each) are copied to shared memory while the first stage runs.
    constexpr int HQC = khat_cols_stride<H>();
    const float* kh0 = wd.khat + (size_t)k * (W / 2 + 1) * HQ;
    float* ksm = col_khat_smem<H, MR>(stw);
    copy_khat<H, NT, NC>(ksm, kh0 + (size_t)(TC * t + c0) * HQ, HQ);
    if constexpr (!CG) grid_wait();
    // the twiddle tables are read after col_chained's first barrier
    col_chained<H, NT, CG, MR, NC>(X, stw, src, wd.conv + k * cplane + (size_t)t * H * TC, ksm,
                                   t == 0 ? kh0 + (size_t)(W / 2) * HQ : nullptr, c0, early);
}

// float2s of a column item's two sequences.
template <int H, int NC = TC>
FFT_CHD constexpr int col_seq_floats2() { return NC * col_stride(H); }

// MR: the radix cap of the build's plans (CMR; 16 for the radix-16 build of sizes whose CMR plan has
// radix 32, launch variant 3)
template <int H, int NT, int MINB, int MR = CMR, int NC = TC>
__global__ void __launch_bounds__(NT, MINB) col_pass(const DevWorld* __restrict__ worlds, const ColItem* __restrict__ items,
                                                const float2* __restrict__ tw, bool early) {
    extern __shared__ float4 smem_raw[];
    float2* X = reinterpret_cast<float2*>(smem_raw);
    float2* stw = X + col_seq_floats2<H, NC>();
    const ColItem it = items[blockIdx.x / (TC / NC)];
    fill_tables<H, MR>(stw, tw, NT);
    col_item<H, NT, false, MR, NC>(worlds[it.world], it, X, stw, NC * (blockIdx.x % (TC / NC)), early);
}

// ------------------------------------------------------------------ paired column pass
// The tile's two spectrum columns as one sequence of cpair elements (re = (c0.re, c1.re),
// im = (c0.im, c1.im)): one thread runs butterfly j of both columns with f32x2 arithmetic and
// 16-byte shared-memory accesses, so the item needs half the threads and about half the
// instructions of the scalar build.  Shared memory: the sequence, the tw2 stage tables, the khat
// columns.
constexpr int PMR = ROW_PLAN;  // largest radix of the paired builds' plans
template <int H>
__device__ __forceinline__ float* col_khat_smem_pair(tw2* stw) {
    constexpr int TWS = tw_table_size(H, PMR);
    return reinterpret_cast<float*>(stw + TWS + 1);
}

// The chained paired item: as col_chained, with one butterfly of both columns per thread (a warp's access
// to the tile is 512 contiguous bytes).
template <int H, int NT>
__device__ __forceinline__ void col_chained_pair(cpair* X, const tw2* stw, const float2* __restrict__ src,
                                                 float2* __restrict__ dst, const float* ksm,
                                                 const float* __restrict__ khn, bool early) {
    constexpr int LAST = plan_len(H, PMR) - 1, R = plan_radix(H, 0, PMR), NB = H / R;
    constexpr int HQC = khat_cols_stride<H>();
    static_assert(fusable<H, PMR>() && NB <= NT, "one outer butterfly per thread");
    const int j = threadIdx.x;
    const bool on = NB == NT || j < NB;
    const tw2* last = stw + stage_tw_offset(H, LAST, PMR);
    cpair v[R];
    if (on) {
        const float4* s4 = reinterpret_cast<const float4*>(src) + j;
        const uint64_t keep = hint::policy_keep();
#pragma unroll
        for (int m = 0; m < R; m++) {
            const float4 q = hint::ld4(s4 + m * NB, keep);
            v[m] = cpair{make_float2(q.x, q.z), make_float2(q.y, q.w)};
        }
        Dft<R, false>::run(v);
        stage_store<H, R, 1>(X, j, v);
    }
    cp_async_wait_all();  // the khat columns
    __syncthreads();
    fft_stages<H, 1, NT, false, 1, LAST>(X, stw);
    if (on) {
        stage_load<H, R, NB, false>(X, j, v, last);
        if (khn == nullptr) {
#pragma unroll
            for (int m = 0; m < R; m++) {
                const int ky = j + m * NB, kk = ky <= H / 2 ? ky : H - ky;
                v[m] = cscale2(v[m], make_float2(ksm[kk], ksm[HQC + kk]));
            }
        }
    }
    if (khn != nullptr) {  // tile 0, see col_chained
        __syncthreads();
        if (on)
#pragma unroll
            for (int m = 0; m < R; m++) X[j + m * NB] = v[m];
        __syncthreads();
        if (on)
#pragma unroll
            for (int m = 0; m < R; m++) {
                const int ky = j + m * NB, kk = ky <= H / 2 ? ky : H - ky;
                const cpair zm = X[(H - ky) % H];
                const float2 p = packed_times_khat(make_float2(v[m].re.x, v[m].im.x), make_float2(zm.re.x, zm.im.x),
                                                   ksm[kk], khn[kk]);
                const float k1 = ksm[HQC + kk];
                v[m] = cpair{make_float2(p.x, v[m].re.y * k1), make_float2(p.y, v[m].im.y * k1)};
            }
    }
    if (on) Dft<R, true>::run(v);
    __syncthreads();
    if (on) stage_store<H, R, 1>(X, j, v);
    __syncthreads();
    if (early) grid_trigger();
    fft_stages<H, 1, NT, true, 1, LAST>(X, stw);
    if (on) {
        stage_load<H, R, NB, true>(X, j, v, last);
        float4* d4 = reinterpret_cast<float4*>(dst) + j;
        const uint64_t keep = hint::policy_keep();
#pragma unroll
        for (int m = 0; m < R; m++) hint::st4(d4 + m * NB, make_float4(v[m].re.x, v[m].im.x, v[m].re.y, v[m].im.y), keep);
    }
}

template <int H, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) col_pass_pair(const DevWorld* __restrict__ worlds,
                                                     const ColItem* __restrict__ items, const float2* __restrict__ tw,
                                                     bool early) {
    extern __shared__ float4 smem_raw[];
    cpair* X = reinterpret_cast<cpair*>(smem_raw);
    tw2* stw = reinterpret_cast<tw2*>(X + seq_stride(H));
    const ColItem it = items[blockIdx.x];
    const DevWorld& wd = worlds[it.world];
    fill_stage_twiddles<H, tw2, 0, PMR>(stw, tw, threadIdx.x, NT);
    const int W = wd.W, c = it.chan, t = it.tile, k = it.kernel, HQ = wd.HQ;
    const size_t cplane = (size_t)(W / 2) * H;
    const float2* src = wd.spec + c * cplane + (size_t)t * H * TC;
    float2* dst = wd.conv + k * cplane + (size_t)t * H * TC;
    const float* kh0 = wd.khat + (size_t)k * (W / 2 + 1) * HQ;
    float* ksm = col_khat_smem_pair<H>(stw);
    copy_khat<H, NT>(ksm, kh0 + (size_t)TC * t * HQ, HQ);
    grid_wait();
    col_chained_pair<H, NT>(X, stw, src, dst, ksm, t == 0 ? kh0 + (size_t)(W / 2) * HQ : nullptr, early);
}

// Sizes built: each TU instantiates one group.  Threads per CTA: one first-stage butterfly per
// thread for the two sequences a CTA holds (2N / outer radix), in whole warps, at most 1024.  (With at least 64
// the columns of 64 to 256 left half of every CTA idle: 1024 worlds of 256 x 256 311 -> 249 us a generation.)
#define LENIA_SIZES_SMALL(X) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(384) X(512) X(768)
#define LENIA_SIZES_LARGE(X) X(1024) X(1536) X(2048) X(3072) X(4096) X(6144) X(8192)
template <int N, int MR = CMR> constexpr int nt_of() {
    // one outer butterfly per thread, two sequences, whole warps
    constexpr int n = (2 * (is_two_stage(N, MR) ? two_tw_len(N) : N / plan_radix(N, 0, MR)) + 31) / 32 * 32;
    return n > 1024 ? 1024 : n;
}
// whether the scalar column build's plan has radix 32 (1024, 8192)
template <int N> constexpr bool col_r32() { return plan_radix(N, 0, CMR) == 32; }
// variant 0: at most 64 registers per thread (80 for radix-32 plans: the 1024 build spilled 508 B at
// 64 and needs none at 80); variant 1: at most 128
template <int N, int V, int MR = CMR> constexpr int minb_threads() {
    return V == 0 ? (plan_radix(N, 0, MR) == 32 || two_stage(N, MR).ra > 16 ? 768 : 1024) : 512;
}
template <int N, int V, int MR = CMR> constexpr int minb_of() {
    return minb_threads<N, V, MR>() / nt_of<N, MR>() < 1 ? 1 : minb_threads<N, V, MR>() / nt_of<N, MR>();
}
// paired column build: one first-stage butterfly per thread for the one (paired) sequence, at most
// 128 registers a thread
template <int N> constexpr int nt_pair_of() {
    constexpr int n = N / plan_radix(N, 0, PMR);
    return n < 64 ? 64 : (n > 1024 ? 1024 : n);
}
template <int N> constexpr int minb_pair_of() { return 512 / nt_pair_of<N>() < 1 ? 1 : 512 / nt_pair_of<N>(); }

// Launch one instantiation.  Dynamic shared memory above 48 KB must be enabled per kernel before
// its first launch and before any stream capture that contains it; a zero-item call does just that.
template <int H, int NT, int MINB, int MR = CMR, int NC = TC>
bool col_go(const DevWorld* worlds, const ColItem* items, int nitems, const float2* tw, LaunchOn s) {
    const size_t smem = col_seq_floats2<H, NC>() * sizeof(float2) + stage_table_bytes<H, MR>() + col_khat_bytes<H>() / (TC / NC) + 16;
    static int attr_max = 0;
    if ((int)smem > attr_max) {
        if (cudaFuncSetAttribute(col_pass<H, NT, MINB, MR, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
            return false;
        attr_max = (int)smem;
    }
    return nitems <= 0 || launch_pass(col_pass<H, NT, MINB, MR, NC>, nitems * (TC / NC), NT, smem, s, worlds, items, tw, s.early);
}

template <int H>
constexpr size_t col_pair_smem() {
    return (size_t)seq_stride(H) * sizeof(cpair) + (size_t)(tw_table_size(H, PMR) + 1) * sizeof(tw2) + col_khat_bytes<H>();
}

template <int H, int NT, int MINB>
bool col_go_pair(const DevWorld* worlds, const ColItem* items, int nitems, const float2* tw, LaunchOn s) {
    const size_t smem = col_pair_smem<H>();
    static int attr_max = 0;
    if ((int)smem > attr_max) {
        if (cudaFuncSetAttribute(col_pass_pair<H, NT, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
            return false;
        attr_max = (int)smem;
    }
    return nitems <= 0 || launch_pass(col_pass_pair<H, NT, MINB>, nitems, NT, smem, s, worlds, items, tw, s.early);
}

// Shared memory of a row-pass launch: sequences (in the general step twice, for a second kernel's sequences or the plane),
// then the stage tables.
template <int W, bool GEN>
constexpr size_t row_smem(int seqs = row_seqs(W, GEN)) {
    return (size_t)(GEN ? 2 : 1) * seqs * seq_stride(W) * sizeof(float2) + stage_table_bytes<W>();
}

template <int W, int V, bool GEN>
bool row_go(int mode, const DevWorld* worlds, const RowItem* items, int nitems, const float2* tw, LaunchOn s) {
    constexpr int S = row_cta_seqs(W, V, GEN), NT = row_nt<W, GEN, V>();
    constexpr auto kernel = row_pass<W, NT, row_minb<W, V, GEN>(), S, GEN, row_wide<W, V>()>;
    const size_t smem = row_smem<W, GEN>(S);
    static int attr_max = 0;
    if ((int)smem > attr_max) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
            return false;
        attr_max = (int)smem;
    }
    return nitems <= 0 || launch_pass(kernel, nitems * (row_seqs(W, GEN) / S), NT, smem, s, worlds, items, mode, tw, s.early);
}

// Column-pass builds: variant 0 and 1 are the scalar build at 64 (80 with a radix-32 plan) and 128
// registers a thread, variant 2 the paired build, variant 3 the scalar build with the radix-16 plan at
// 64 registers where the scalar plan has radix 32 and the sides are below 2048, from 2048 up the
// scalar build with one column a CTA (elsewhere variant 0).
template <int N>
bool col_go_variant(int variant, const DevWorld* worlds, const ColItem* items, int nitems, const float2* tw,
                    LaunchOn s) {
    if (variant == 2) return col_go_pair<N, nt_pair_of<N>(), minb_pair_of<N>()>(worlds, items, nitems, tw, s);
    if (variant == 1) return col_go<N, nt_of<N>(), minb_of<N, 1>()>(worlds, items, nitems, tw, s);
    if constexpr (N >= 2048) {
        if (variant == 3)
            return col_go<N, nt_of<N>() / TC, minb_threads<N, N == 8192>() / (nt_of<N>() / TC), CMR, 1>(worlds, items, nitems, tw, s);
    } else if constexpr (col_r32<N>()) {
        if (variant == 3) return col_go<N, nt_of<N, 16>(), minb_of<N, 0, 16>(), 16>(worlds, items, nitems, tw, s);
    }
    return col_go<N, nt_of<N>(), minb_of<N, 0>()>(worlds, items, nitems, tw, s);
}
#define LENIA_COL_CASE(N) \
    case N: return col_go_variant<N>(variant, worlds, items, nitems, tw, s);

// Row-pass builds: variant bit 0 selects the register cap (row_minb); the single-kernel (GEN =
// false) and general (GEN = true) builds sit in separate translation units, which keeps each
// unit's compile time down.  (A paired row build, two packed sequences per thread as in the
// column pass, measured 15% slower at 4096 x 4096: its stores and growth had half the warps to
// hide behind.)
#define LENIA_ROW_CASE_G(N, G)                                                                     \
    case N:                                                                                        \
        return (variant & 1) ? row_go<N, 1, G>(mode, worlds, items, nitems, tw, s) \
                             : row_go<N, 0, G>(mode, worlds, items, nitems, tw, s);
#define LENIA_ROW_CASE_SIMPLE(N) LENIA_ROW_CASE_G(N, false)
#define LENIA_ROW_CASE_GENERAL(N) LENIA_ROW_CASE_G(N, true)

bool launch_col_group_small(int H, int variant, const DevWorld* worlds, const ColItem* items, int nitems,
                            const float2* tw, LaunchOn s);
bool launch_col_group_large(int H, int variant, const DevWorld* worlds, const ColItem* items, int nitems,
                            const float2* tw, LaunchOn s);
#define LENIA_ROW_GROUP_DECL(NAME)                                                                       \
    bool NAME(int W, int variant, int mode, const DevWorld* worlds, const RowItem* items, \
              int nitems, const float2* tw, LaunchOn s);
LENIA_ROW_GROUP_DECL(launch_row_group_small_simple)
LENIA_ROW_GROUP_DECL(launch_row_group_small_general)
LENIA_ROW_GROUP_DECL(launch_row_group_large_simple)
LENIA_ROW_GROUP_DECL(launch_row_group_large_general)

}  // namespace lenia
