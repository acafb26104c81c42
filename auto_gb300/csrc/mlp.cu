// The learned screen proposer: a 16 -> 256 -> 256 -> 3 MLP in BF16 with FP32 accumulation,
// trained by hand-written forward and backward kernels.
//
// It predicts, from a world's kernel and growth parameters, P(survives), P(moves), P(explodes);
// the batched simulator generates the labels and remains the judge of every proposed world.  The
// reference has no learned component; its world screen samples parameters uniformly
// (scripts/life_screen.py:143-179), which is the baseline this proposer is compared with.
//
// Parameters: FP32 master weights updated by Adam; BF16 copies feed every GEMM; activations are
// rounded to BF16; every GEMM accumulates in FP32.  The GEMMs of the two 256-wide layers -- forward h1
// and h2, backward dh1 and the weight gradients dW1 and dW2 -- run on the 5th-generation tensor cores
// (tcgen05 MMAs, TMEM accumulators), the 3-wide output layer in the hand-overs between them, all in
// one kernel (mlp_tile) that keeps a tile's activations in shared memory.
//   layer 1: W1 [256 x 16],  b1 [256]      h1 = relu(x W1^T + b1)
//   layer 2: W2 [256 x 256], b2 [256]      h2 = relu(h1 W2^T + b2)
//   layer 3: W3 [3 x 256],   b3 [3]        z  = h2 W3^T + b3,  p = sigmoid(z)
//   loss: mean over the batch and the 3 labels of softplus(z) - y z  (binary cross-entropy)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "engine.cuh"
#include "tc_ptx.cuh"

namespace lenia {
namespace mlp {

constexpr int IN = 16, HID = 256, OUT = 3;
constexpr int P_W1 = 0, P_B1 = P_W1 + HID * IN, P_W2 = P_B1 + HID, P_B2 = P_W2 + HID * HID, P_W3 = P_B2 + HID,
              P_B3 = P_W3 + OUT * HID, NPARAM = P_B3 + OUT;

using bf16 = __nv_bfloat16;

// ------------------------------------------------------------------ the network on a tile of rows
// One CTA takes 128 rows through the whole network, forward to the logits and back to every gradient.
// Nothing but the inputs, the weights and the results touches global memory.
//
// All operands sit in shared memory in the canonical layout without swizzle (8-row x 16-byte core
// matrices, K-adjacent ones 128 bytes apart, 8-row groups one after another: tc::kmajor_offset).  A
// matrix stored [r][c] that way is a K-major operand with K = c (LBO 128, SBO one row group) and, read
// with the roles exchanged, an MN-major operand with K = r (LBO one row group, SBO 128): the same bytes
// serve h1, dh2, dh1 and W2 in both of their products, so nothing is transposed or stored twice.
//
//   D      = x W1^T                       A x [m][i]        B W1 [o][i]      N = 256, K = 16
//   h1     = relu(D + b1)                 -> R2
//   D      = h1 W2^T                      A h1              B W2 [o][i]      N = 256, K = 256
//   h2     = relu(D + b2), z = h2 W3^T + b3                                  (CUDA cores, per row)
//   dz     = (sigmoid(z) - y) / (3 B), dh2 = (dz W3) * (h2 > 0) -> R1
//   D      = dh2 W2                       A dh2             B W2 (MN-major)  N = 256, K = 256
//   dh1    = D * (h1 > 0)                 -> R0
//   dW2   += dh2^T h1                     A dh2 (MN-major)  B h1 (MN-major)  M = 2 x 128, N = 256, K = 128 rows
//   dW1   += dh1^T x                      A dh1 (MN-major)  B x (MN-major)   M = 2 x 128, N = 16,  K = 128 rows
//
// The bias gradients are column sums of the unrounded FP32 dh2 and dh1 (transposed by shuffles), dW3
// of dz h2; weight gradients of several tiles meet in global memory with vector reductions.  512
// threads: warp w reads TMEM lanes 32 (w % 4) .. + 31 (the tile's rows) and columns 64 (w / 4) .. + 63.
//
// W2 takes R0 and R1 (128 KB); the backward pass needs R1 for dh2 and fetches W2's rows 128..255
// again into R0.  One CTA per SM (224 KB of shared memory, all 512 TMEM columns).  A tile is a chain of
// five waits on the tensor cores with a hand-over after each, so it is bound by that latency, and a batch of
// 1000 rows by one tile's: with a thread for every 64 columns of a row instead of every 128,
// lenia_mlp_gradients of 1000 rows went from 77 to 66 us; with the gradient reductions on whole 128-byte runs
// (transpose_pieces) lenia_mlp_train_step of 1000 rows from 57.8 to 55.4, of 4096 from 60.1 to 57.5.  As separate
// GEMM launches, whose hand-overs wrote h1 and h2 (and their transposes) to global memory with 2-byte stores one
// row stride apart per lane, the gradients took 560.
//
// Every barrier wait is bounded; a CTA that gives up waits (bounded) for its MMAs and copies, raises *err,
// frees its TMEM and returns.
constexpr int TILE = 128, NTHR = 512, NCOL = TILE * HID / NTHR;  // columns of a row per thread
constexpr uint32_t GROUP = HID * 2 * 8;    // bytes of eight 256-wide rows
constexpr uint32_t XGROUP = IN * 2 * 8;    // bytes of eight 16-wide rows
constexpr uint32_t REGION = TILE * HID * 2;  // 64 KB
constexpr uint32_t S_W1 = 3 * REGION, S_X = S_W1 + HID * IN * 2, S_F = S_X + TILE * IN * 2;
// floats from S_F: b1, b2, W3, the other column quarters' logits (then dz), and the sums db2, db1, dW3, db3
constexpr int F_B1 = 0, F_B2 = F_B1 + HID, F_W3 = F_B2 + HID, F_Z = F_W3 + OUT * HID, F_DB2 = F_Z + (HID / NCOL - 1) * TILE * OUT,
              F_DB1 = F_DB2 + HID, F_DW3 = F_DB1 + HID, F_DB3 = F_DW3 + OUT * HID, F_END = F_DB3 + 4;
constexpr uint32_t S_BAR = S_F + F_END * 4;
constexpr uint32_t TILE_SMEM = S_BAR + 16;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint4 pack8(const float* v) {
    return make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
}
// Sums of 32 per-lane values over the warp's lanes: lane l gets the sum of the lanes' v[l] (each
// step folds half of the remaining columns onto the other half's lanes).
__device__ __forceinline__ float column_sums(float* v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
#pragma unroll
        for (int i = 0; i < w; i++) {
            const bool up = lane & w;
            const float send = up ? v[i] : v[i + w], keep = up ? v[i + w] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
    }
    return v[0];
}

// Eight lanes' eight float4s each (v[4 i ..]: piece i of a row) transposed among them: lane l of eight then holds
// piece l of rows 0..7 in v[4 r ..].
__device__ __forceinline__ void transpose_pieces(float* v) {
#pragma unroll
    for (int w = 4; w >= 1; w >>= 1) {
        const bool up = threadIdx.x & w;
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (!(i & w))
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    float &lo = v[4 * i + k], &hi = v[4 * (i + w) + k];
                    const float got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, w);
                    if (up) lo = got;
                    else hi = got;
                }
    }
}

// rows [first, first + n) of W2 (bf16 [256][256]) into an operand region, n a multiple of 8: eight rows of
// one 16-byte column piece per eight lanes, 128 contiguous bytes of shared memory
template <int NT = NTHR>
__device__ __forceinline__ void load_w2(uint8_t* dst, const bf16* __restrict__ w2, int first, int n) {
    for (int e = threadIdx.x; e < n * (HID / 8); e += NT) {
        const int r = (e >> 8) * 8 + (e & 7), kg = (e >> 3) & 31;
        cp_async16(dst + tc::kmajor_offset(r, 8 * kg, HID, 2), w2 + (size_t)(first + r) * HID + 8 * kg);
    }
}

__global__ void __launch_bounds__(NTHR, 1)
    mlp_tile(const float* __restrict__ x, const float* __restrict__ y, int B, const float* __restrict__ w,
             const bf16* __restrict__ wb, float* __restrict__ g, float* __restrict__ loss_rows, int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t *R0 = sm, *R1 = sm + REGION, *R2 = sm + 2 * REGION, *W1s = sm + S_W1, *Xs = sm + S_X;
    float* F = reinterpret_cast<float*>(sm + S_F);
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + S_BAR);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = (warp & 3) * 32 + lane, part = warp >> 2;  // this thread's tile row and column quarter
    const int ntiles = (B + TILE - 1) / TILE;
    const bf16* w2 = wb + P_W2;

    for (int e = tid; e < HID * 2; e += NTHR)
        cp_async16(W1s + tc::kmajor_offset(e >> 1, 8 * (e & 1), IN, 2), wb + P_W1 + (e >> 1) * IN + 8 * (e & 1));
    asm volatile("cp.async.commit_group;" ::: "memory");
    load_w2(R0, w2, 0, HID);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int e = tid; e < HID; e += NTHR) F[F_B1 + e] = w[P_B1 + e], F[F_B2 + e] = w[P_B2 + e];
    for (int e = tid; e < OUT * HID; e += NTHR) F[F_W3 + e] = __bfloat162float(wb[P_W3 + e]);
    for (int e = F_DB2 + tid; e < F_END; e += NTHR) F[e] = 0.f;
    if (tid == 0) {
        tc::mbar_init(bar, 1);
        tc::fence_barrier_init();
    }
    if (warp == 0) tc::tmem_alloc(slot, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *slot, mine = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t r0 = tc::smem_u32(R0), r1 = tc::smem_u32(R1), r2 = tc::smem_u32(R2), xs = tc::smem_u32(Xs),
                   w1s = tc::smem_u32(W1s);
    constexpr uint32_t ID_FWD = tc::instr_desc(1, 128, HID), ID_DH1 = tc::instr_desc(1, 128, HID, false, true),
                       ID_DW2 = tc::instr_desc(1, 128, HID, true, true), ID_DW1 = tc::instr_desc(1, 128, IN, true, true);

    uint32_t phase = 0;
    bool pending = false;  // a commit that no wait has seen (uniform across the CTA)
    auto commit = [&]() {  // thread 0
        tc::mma_commit(bar);
    };
    // wait for the last commit; false (for the whole CTA) if it did not come
    auto wait = [&]() -> bool {
        const bool gave_up = __syncthreads_or(!tc::mbar_wait(bar, phase));
        phase ^= 1;
        pending = gave_up;
        tc::tc_fence_after();
        return !gave_up;
    };
    // shared-memory operands written and TMEM read: thread 0 may issue MMAs
    auto publish = [&]() {
        tc::tc_fence_before();
        tc::fence_async_smem();
        __syncthreads();
        tc::tc_fence_after();
    };

    // eight inputs of a tile for each of the first 256 threads: row tid / 2, half a row each
    float xin[8];
    const bool loads = tid < 2 * TILE;
    auto fetch = [&](int t) {
        const int r = t * TILE + (tid >> 1);
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (loads && r < B) {
            const float4* p = reinterpret_cast<const float4*>(x + (size_t)r * IN + 8 * (tid & 1));
            a = p[0], b = p[1];
        }
        xin[0] = a.x, xin[1] = a.y, xin[2] = a.z, xin[3] = a.w, xin[4] = b.x, xin[5] = b.y, xin[6] = b.z, xin[7] = b.w;
    };
    bool ok = true, first = true;
    fetch(blockIdx.x);
    for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, first = false) {
        if (!first) load_w2(R0, w2, 0, HID);  // the backward pass of the last tile took its place
        if (loads) *reinterpret_cast<uint4*>(Xs + tc::kmajor_offset(tid >> 1, 8 * (tid & 1), IN, 2)) = pack8(xin);
        if (first) asm volatile("cp.async.wait_group 1;" ::: "memory");  // W1
        publish();
        if (tid == 0) {
            tc::mma<false>(tmem, tc::smem_desc(xs, 128, XGROUP), tc::smem_desc(w1s, 128, XGROUP), ID_FWD, 0u);
            commit();
        }
        pending = true;
        if (t + (int)gridDim.x < ntiles) fetch(t + gridDim.x);
        if (!(ok = wait())) break;
        // rows past the batch are zeros in every product (a row that is not there meets no infinite weight)
        const int b = t * TILE + row;
        const bool valid = b < B;
        float yy[OUT] = {0.f, 0.f, 0.f};  // labels, wanted after the second layer
        if (part == 0 && valid)
#pragma unroll
            for (int o = 0; o < OUT; o++) yy[o] = y[(size_t)b * OUT + o];
#pragma unroll
        for (int c = 0; c < NCOL / 32; c++) {
            const int n0 = part * NCOL + 32 * c;
            float v[32];
            tc::tmem_ld32(mine + n0, v);
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = valid ? fmaxf(v[i] + F[F_B1 + n0 + i], 0.f) : 0.f;
#pragma unroll
            for (int i = 0; i < 4; i++)
                *reinterpret_cast<uint4*>(R2 + tc::kmajor_offset(row, n0 + 8 * i, HID, 2)) = pack8(v + 8 * i);
        }
        cp_async_wait0();  // W2
        publish();
        if (tid == 0) {
            for (uint32_t s = 0; s < HID / 16; s++)
                tc::mma<false>(tmem + HID, tc::smem_desc(r2 + 256u * s, 128, GROUP), tc::smem_desc(r0 + 256u * s, 128, GROUP),
                               ID_FWD, s > 0);
            commit();
        }
        pending = true;
        if (!(ok = wait())) break;
        float z[OUT] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < NCOL / 32; c++) {
            const int n0 = part * NCOL + 32 * c;
            float v[32];
            tc::tmem_ld32(mine + HID + n0, v);
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const float h = __bfloat162float(__float2bfloat16_rn(fmaxf(v[i] + F[F_B2 + n0 + i], 0.f)));
#pragma unroll
                for (int o = 0; o < OUT; o++) z[o] = fmaf(h, F[F_W3 + o * HID + n0 + i], z[o]);
            }
        }
        if (part > 0)
            for (int o = 0; o < OUT; o++) F[F_Z + ((part - 1) * TILE + row) * OUT + o] = z[o];
        tc::tc_fence_before();
        __syncthreads();
        tc::tc_fence_after();
        if (part == 0) {
            float l = 0.f, dz[OUT];
#pragma unroll
            for (int o = 0; o < OUT; o++) {
                float zz = z[o];
                for (int q = 0; q < HID / NCOL - 1; q++) zz += F[F_Z + (q * TILE + row) * OUT + o];
                zz += w[P_B3 + o];
                const float p = 1.f / (1.f + expf(-zz));
                l += fmaxf(zz, 0.f) - zz * yy[o] + log1pf(expf(-fabsf(zz)));
                dz[o] = valid ? (p - yy[o]) / (float)(B * OUT) : 0.f;
                F[F_Z + row * OUT + o] = __bfloat162float(__float2bfloat16_rn(dz[o]));
            }
            if (valid) loss_rows[b] = l / OUT;
#pragma unroll
            for (int o = 0; o < OUT; o++) {
                for (int d = 16; d > 0; d >>= 1) dz[o] += __shfl_xor_sync(0xffffffffu, dz[o], d);
                if (lane == 0) atomicAdd(&F[F_DB3 + o], dz[o]);
            }
        }
        __syncthreads();
        float dzb[OUT];
        for (int o = 0; o < OUT; o++) dzb[o] = F[F_Z + row * OUT + o];
#pragma unroll 1
        for (int c = 0; c < NCOL / 32; c++) {
            const int n0 = part * NCOL + 32 * c;
            float v[32], q[32];
            tc::tmem_ld32(mine + HID + n0, v);
#pragma unroll
            for (int i = 0; i < 32; i++)
                v[i] = valid ? __bfloat162float(__float2bfloat16_rn(fmaxf(v[i] + F[F_B2 + n0 + i], 0.f))) : 0.f;
#pragma unroll
            for (int o = 0; o < OUT; o++) {
#pragma unroll
                for (int i = 0; i < 32; i++) q[i] = dzb[o] * v[i];
                atomicAdd(&F[F_DW3 + o * HID + n0 + lane], column_sums(q));
            }
#pragma unroll
            for (int i = 0; i < 32; i++) {
                float d = 0.f;
#pragma unroll
                for (int o = 0; o < OUT; o++) d = fmaf(dzb[o], F[F_W3 + o * HID + n0 + i], d);
                v[i] = v[i] > 0.f ? d : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
                *reinterpret_cast<uint4*>(R1 + tc::kmajor_offset(row, n0 + 8 * i, HID, 2)) = pack8(v + 8 * i);
            atomicAdd(&F[F_DB2 + n0 + lane], column_sums(v));
        }
        publish();
        if (tid == 0) {
            for (uint32_t s = 0; s < 8; s++)
                tc::mma<false>(tmem, tc::smem_desc(r1 + 256u * s, 128, GROUP), tc::smem_desc(r0 + 2 * GROUP * s, GROUP, 128),
                               ID_DH1, s > 0);
            commit();
        }
        pending = true;
        if (!(ok = wait())) break;
        load_w2(R0, w2, 128, 128);
        cp_async_wait0();
        publish();
        if (tid == 0) {
            for (uint32_t s = 0; s < 8; s++)
                tc::mma<false>(tmem, tc::smem_desc(r1 + 256u * (8 + s), 128, GROUP),
                               tc::smem_desc(r0 + 2 * GROUP * s, GROUP, 128), ID_DH1, 1u);
            for (uint32_t s = 0; s < 8; s++)  // dW2, outputs 128..255
                tc::mma<false>(tmem + HID, tc::smem_desc(r1 + 16 * 128 + 2 * GROUP * s, GROUP, 128),
                               tc::smem_desc(r2 + 2 * GROUP * s, GROUP, 128), ID_DW2, s > 0);
            commit();
        }
        pending = true;
        if (!(ok = wait())) break;
#pragma unroll 1
        for (int c = 0; c < NCOL / 32; c++) {
            const int n0 = part * NCOL + 32 * c;
            float v[32];
            tc::tmem_ld32(mine + n0, v);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 h = *reinterpret_cast<const uint4*>(R2 + tc::kmajor_offset(row, n0 + 8 * i, HID, 2));
                const uint32_t hw[4] = {h.x, h.y, h.z, h.w};
                // h1 is a ReLU's output: zero where its bits (sign aside) are
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (((hw[k / 2] >> (16 * (k & 1))) & 0x7fffu) == 0u) v[8 * i + k] = 0.f;
                *reinterpret_cast<uint4*>(R0 + tc::kmajor_offset(row, n0 + 8 * i, HID, 2)) = pack8(v + 8 * i);
            }
            atomicAdd(&F[F_DB1 + n0 + lane], column_sums(v));
        }
        publish();
        if (tid == 0) {
            for (uint32_t s = 0; s < 8; s++)  // dW2, outputs 0..127
                tc::mma<false>(tmem, tc::smem_desc(r1 + 2 * GROUP * s, GROUP, 128),
                               tc::smem_desc(r2 + 2 * GROUP * s, GROUP, 128), ID_DW2, s > 0);
            commit();
        }
        pending = true;
        auto add_dw2 = [&](uint32_t col0, int out0) {
#pragma unroll 1
            for (int c = 0; c < NCOL / 32; c++) {
                const int n0 = part * NCOL + 32 * c;
                float v[32];
                tc::tmem_ld32(mine + col0 + n0, v);
                // eight lanes on 128 contiguous bytes of a row instead of 32 lanes on 32 rows
                transpose_pieces(v);
                float* p = g + P_W2 + (size_t)(out0 + (row & ~7)) * HID + n0 + 4 * (lane & 7);
#pragma unroll
                for (int r = 0; r < 8; r++) red_add4(p + r * HID, v[4 * r], v[4 * r + 1], v[4 * r + 2], v[4 * r + 3]);
            }
        };
        add_dw2(HID, 128);
        if (!(ok = wait())) break;
        publish();  // the second accumulator is read
        if (tid == 0) {
            for (uint32_t m = 0; m < 2; m++)
                for (uint32_t s = 0; s < 8; s++)
                    tc::mma<false>(tmem + HID + IN * m, tc::smem_desc(r0 + 16 * 128 * m + 2 * GROUP * s, GROUP, 128),
                                   tc::smem_desc(xs + 2 * XGROUP * s, XGROUP, 128), ID_DW1, s > 0);
            commit();
        }
        pending = true;
        add_dw2(0, 0);
        if (!(ok = wait())) break;
        if (part < 2) {
            float v[16];  // part p: units 128 p + row
            tc::tmem_ld16(mine + HID + IN * part, v);
            float* p = g + P_W1 + (size_t)(128 * part + row) * IN;
#pragma unroll
            for (int i = 0; i < 16; i += 4) red_add4(p + i, v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
        tc::tc_fence_before();
        __syncthreads();
        tc::tc_fence_after();
    }
    cp_async_wait0();
    __syncthreads();
    if (ok && (int)blockIdx.x < ntiles) {
        for (int e = tid; e < HID; e += NTHR) {
            atomicAdd(g + P_B2 + e, F[F_DB2 + e]);
            atomicAdd(g + P_B1 + e, F[F_DB1 + e]);
        }
        for (int e = tid; e < OUT * HID; e += NTHR) atomicAdd(g + P_W3 + e, F[F_DW3 + e]);
        if (tid < OUT) atomicAdd(g + P_B3 + tid, F[F_DB3 + tid]);
    }
    if (!ok && tid == 0) {
        if (pending) tc::mbar_wait(bar, phase ^ 1);  // drain the commit that did not come in time, bounded
        *(volatile int*)err = 1;
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

// ------------------------------------------------------------------ ranking: the forward pass alone
// The same tile and operands as mlp_tile, as a pipeline of two groups of eight warps.  Group A takes a tile through the
// first layer (x W1^T, then h1 into R2) and issues the second layer's MMAs; group B takes the second layer's accumulator to
// the probabilities.  A works on tile t + 1 while B works on tile t: h1 may be overwritten once the
// second layer's MMAs of tile t have completed (bar2), its accumulator once B has read it (free2).
// lenia_mlp_predict of 250001 rows: 11.1 ms as separate GEMM launches of 4096 rows, 372 us with one group running a tile's
// hand-overs one after the other and copied inputs, 336 with two groups, 175 with the inputs read in place (in_place).
// A wait that gives up ends its own group, and the other group's next wait gives up in turn.
constexpr int NGROUP = 256, NRANK = 2 * NGROUP;
constexpr uint32_t RANK_SMEM = S_BAR + 32;
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

__global__ void __launch_bounds__(NRANK, 1)
    mlp_rank(const float* __restrict__ x, int B, const float* __restrict__ w, const bf16* __restrict__ wb,
             float* __restrict__ probs, int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t *R0 = sm, *R2 = sm + 2 * REGION, *W1s = sm + S_W1, *Xs = sm + S_X;
    float* F = reinterpret_cast<float*>(sm + S_F);
    uint64_t *bar1 = reinterpret_cast<uint64_t*>(sm + S_BAR), *bar2 = bar1 + 1, *free2 = bar1 + 2;
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar1 + 3);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = (warp & 3) * 32 + lane, half = (warp >> 2) & 1;
    const int ntiles = (B + TILE - 1) / TILE;
    const bf16* w2 = wb + P_W2;

    for (int e = tid; e < HID * 2; e += NRANK)
        cp_async16(W1s + tc::kmajor_offset(e >> 1, 8 * (e & 1), IN, 2), wb + P_W1 + (e >> 1) * IN + 8 * (e & 1));
    asm volatile("cp.async.commit_group;" ::: "memory");
    load_w2<NRANK>(R0, w2, 0, HID);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int e = tid; e < HID; e += NRANK) F[F_B1 + e] = w[P_B1 + e], F[F_B2 + e] = w[P_B2 + e];
    for (int e = tid; e < OUT * HID; e += NRANK) F[F_W3 + e] = __bfloat162float(wb[P_W3 + e]);
    if (tid == 0) {
        tc::mbar_init(bar1, 1);
        tc::mbar_init(bar2, 1);
        tc::mbar_init(free2, NGROUP);
        tc::fence_barrier_init();
    }
    if (warp == 0) tc::tmem_alloc(slot, 512);
    asm volatile("cp.async.wait_all;" ::: "memory");
    tc::fence_async_smem();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *slot, mine = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t r0 = tc::smem_u32(R0), r2 = tc::smem_u32(R2), xs = tc::smem_u32(Xs), w1s = tc::smem_u32(W1s);
    constexpr uint32_t IDESC = tc::instr_desc(1, 128, HID);
    const int group = warp >> 3;  // A: 0, B: 1
    // a wait of the whole group (its barrier: 1 + group)
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        const bool ok = !tc::named_sync_or(1 + group, NGROUP, !tc::mbar_wait(bar, parity));
        tc::tc_fence_after();
        return ok;
    };
    bool ok = true;
    uint32_t n = 0;  // tiles this group has begun
    uint32_t issued2 = 0;
    if (group == 0) {
        const int r = tid >> 1, kg = tid & 1;  // this thread's eight inputs of a tile
        float xin[8];
        auto fetch = [&](int t) {
            const int g = t * TILE + r;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (g < B) {
                const float4* p = reinterpret_cast<const float4*>(x + (size_t)g * IN + 8 * kg);
                a = p[0], b = p[1];
            }
            xin[0] = a.x, xin[1] = a.y, xin[2] = a.z, xin[3] = a.w, xin[4] = b.x, xin[5] = b.y, xin[6] = b.z, xin[7] = b.w;
        };
        auto publish = [&]() {
            tc::tc_fence_before();
            tc::fence_async_smem();
            tc::named_sync(1, NGROUP);
            tc::tc_fence_after();
        };
        fetch(blockIdx.x);
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, n++) {
            *reinterpret_cast<uint4*>(Xs + tc::kmajor_offset(r, 8 * kg, IN, 2)) = pack8(xin);
            publish();
            if (tid == 0) {
                tc::mma<false>(tmem, tc::smem_desc(xs, 128, XGROUP), tc::smem_desc(w1s, 128, XGROUP), IDESC, 0u);
                tc::mma_commit(bar1);
            }
            if (t + (int)gridDim.x < ntiles) fetch(t + gridDim.x);
            if (!(ok = wait(bar1, n & 1))) break;
            if (n > 0 && !(ok = wait(bar2, (n - 1) & 1))) break;  // h1 of the last tile has been read
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int n0 = half * 128 + 32 * c;
                float v[32];
                tc::tmem_ld32(mine + n0, v);
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] = fmaxf(v[i] + F[F_B1 + n0 + i], 0.f);
#pragma unroll
                for (int i = 0; i < 4; i++)
                    *reinterpret_cast<uint4*>(R2 + tc::kmajor_offset(row, n0 + 8 * i, HID, 2)) = pack8(v + 8 * i);
            }
            if (n > 0 && !(ok = wait(free2, (n - 1) & 1))) break;  // the last tile's accumulator has been read
            publish();
            if (tid == 0) {
                for (uint32_t s = 0; s < HID / 16; s++)
                    tc::mma<false>(tmem + HID, tc::smem_desc(r2 + 256u * s, 128, GROUP), tc::smem_desc(r0 + 256u * s, 128, GROUP),
                                   IDESC, s > 0);
                tc::mma_commit(bar2);
            }
            issued2 = n + 1;
        }
        // the CTA's last MMAs: waited for by B, and here before TMEM is freed
        if (issued2 > 0 && tid == 0) tc::mbar_wait(bar2, (issued2 - 1) & 1);
        if (!ok && tid == 0) tc::mbar_wait(bar1, n & 1);
    } else {
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, n++) {
            if (!(ok = wait(bar2, n & 1))) break;
            float z[OUT] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int n0 = half * 128 + 32 * c;
                float v[32];
                tc::tmem_ld32(mine + HID + n0, v);
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    const float h = __bfloat162float(__float2bfloat16_rn(fmaxf(v[i] + F[F_B2 + n0 + i], 0.f)));
#pragma unroll
                    for (int o = 0; o < OUT; o++) z[o] = fmaf(h, F[F_W3 + o * HID + n0 + i], z[o]);
                }
            }
            if (half == 1)
                for (int o = 0; o < OUT; o++) F[F_Z + row * OUT + o] = z[o];
            tc::named_sync(2, NGROUP);
            const int b = t * TILE + row;
            if (half == 0) {
#pragma unroll
                for (int o = 0; o < OUT; o++) z[o] += F[F_Z + row * OUT + o];
            }
            tc::tc_fence_before();
            mbar_arrive(free2);
            if (half == 0 && b < B) {
#pragma unroll
                for (int o = 0; o < OUT; o++) probs[(size_t)b * OUT + o] = 1.f / (1.f + expf(-(z[o] + w[P_B3 + o])));
            }
        }
    }
    if (!ok) *(volatile int*)err = 1;
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

__global__ void to_bf16(const float* __restrict__ x, bf16* __restrict__ y, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

__global__ void copy_out(const float* __restrict__ x, float* __restrict__ y, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = x[i];
}

// Adam on the FP32 master weights, refreshing their BF16 copies.
__global__ void adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                     bf16* __restrict__ wb, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    wb[i] = __float2bfloat16_rn(wi);
}

}  // namespace mlp
}  // namespace lenia

using namespace lenia;
using namespace lenia::mlp;

struct LeniaMlp {
    int max_batch = 0;
    int t = 0, sms = 0;
    int reads_host = 0;  // whether kernels may read pageable host memory in place
    cudaStream_t stream = nullptr;
    float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // FP32 master, grads, Adam moments
    bf16* wb = nullptr;                                             // BF16 copy of the parameters
    float *x = nullptr, *y = nullptr, *loss = nullptr;  // a batch: inputs, labels, per-row losses
    int* err = nullptr;  // set by a tile that gave up waiting on a barrier; page-locked host memory, the losses after it
    // ranking: two halves of PREDICT_ROWS rows of inputs and probabilities, each on a stream of its own
    cudaStream_t ps[2] = {};
    float *px = nullptr, *pp = nullptr;
    std::vector<void*> allocs;
};

namespace {

template <typename T>
bool mal(LeniaMlp* n, T** p, size_t count) {
    void* v = nullptr;
    if (cudaMalloc(&v, count * sizeof(T)) != cudaSuccess) return false;
    n->allocs.push_back(v);
    *p = (T*)v;
    return true;
}

int err(const char* msg) {
    cudaGetLastError();  // reported here, and by no later call
    set_thread_error(msg);
    return LENIA_ECUDA;
}

// An error after work has been queued: waits for it first, for kernels and copies of the call may still be reading or
// writing the caller's memory.
int abandon(LeniaMlp* n, const char* msg) {
    for (cudaStream_t s : {n->stream, n->ps[0], n->ps[1]}) cudaStreamSynchronize(s);
    *n->err = 0;
    return err(msg);
}

// rows of inputs that lenia_mlp_predict has on the device at a time, in two halves: a copy of one half
// overlaps the other's tiles.  A half is two tiles for each of the GPU's 152 SMs, about as long on the SMs as on the
// host link.
constexpr int PREDICT_ROWS = 2 * 2 * 152 * TILE;
constexpr uint32_t HALF = PREDICT_ROWS / 2;
// rows of one launch where the kernel reads them in host memory
constexpr int DIRECT_ROWS = 1 << 20;

int tiles_grid(const LeniaMlp* n, int B) {
    const int t = (B + TILE - 1) / TILE;
    return t < n->sms ? t : n->sms;
}

// gradients of the mean BCE of the batch (x, y on the device, or in host memory in_place) into n->g; per-row losses
// into n->loss
bool gradients(LeniaMlp* n, const float* x, const float* y, int B) {
    return cudaMemsetAsync(n->g, 0, (size_t)NPARAM * sizeof(float), n->stream) == cudaSuccess &&
           launch_pass(mlp_tile, tiles_grid(n, B), NTHR, TILE_SMEM, n->stream, x, y, B, n->w, n->wb, n->g, n->loss, n->err);
}

// probabilities of B rows on s (x, probs on the device, or in host memory in_place)
bool rank(LeniaMlp* n, cudaStream_t s, const float* x, uint32_t B, float* probs) {
    return launch_pass(mlp_rank, tiles_grid(n, (int)B), NRANK, RANK_SMEM, s, x, (int)B, n->w, n->wb, probs, n->err);
}

// a kernel with a thread for every parameter
template <class... P, class... A>
bool each_param(LeniaMlp* n, void (*kernel)(P...), A... args) {
    return launch_pass(kernel, (NPARAM + 255) / 256, 256, 0, n->stream, args...);
}

// After the streams have been waited for.
int check_err(LeniaMlp* n) {
    volatile int* flag = n->err;
    if (*flag) {
        *flag = 0;
        return err("mlp: a tile gave up waiting on a barrier; results are invalid");
    }
    return 0;
}

// Whether a kernel may read host rows where they are: the GPU walks the host's page tables (Grace), the rows are aligned
// for its loads (16 bytes, labels 4), and they are the host's (device memory is no valid argument and stays with the copy).
// Against copying them first, lenia_mlp_predict of 250001 rows 336 -> 188 us, of 1000 rows 50 -> 42, lenia_mlp_gradients of
// 1000 rows 84 -> 72.
bool in_place(const LeniaMlp* n, const float* rows, uintptr_t align = 16) {
    if (!n->reads_host || (uintptr_t)rows % align) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, rows) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeDevice;
}

// Reads a word of every page of a range that a kernel will read in place (touch_pages): a page that is not the caller's faults
// on the host, and one that is not there yet gets its place from it.  256 pages of 64 KB for 250001 rows.
void touch_rows(const float* p, size_t count) { touch_pages(const_cast<float*>(p), count * sizeof(float), false); }

// The batch's gradients from host rows, copied first where they cannot be read in place.
int batch_gradients(LeniaMlp* n, const float* x, const float* y, uint32_t B) {
    if (!in_place(n, x) || !in_place(n, y, 4)) {
        if (cudaMemcpyAsync(n->x, x, (size_t)B * IN * 4, cudaMemcpyHostToDevice, n->stream) != cudaSuccess ||
            cudaMemcpyAsync(n->y, y, (size_t)B * OUT * 4, cudaMemcpyHostToDevice, n->stream) != cudaSuccess)
            return abandon(n, "mlp: upload failed");
        x = n->x, y = n->y;
    } else {
        touch_rows(x, (size_t)B * IN);
        touch_rows(y, (size_t)B * OUT);
    }
    return gradients(n, x, y, (int)B) ? 0 : abandon(n, "mlp: launch failed");
}

// Waits for the batch; its mean loss.
int mean_loss(LeniaMlp* n, uint32_t B, float* loss) {
    if (cudaStreamSynchronize(n->stream) != cudaSuccess) return abandon(n, "mlp: the batch failed");
    double s = 0;
    for (uint32_t i = 0; i < B; i++) s += n->loss[i];
    if (loss) *loss = (float)(s / B);
    return check_err(n);
}

// Probabilities of count rows.  A chunk's may leave before the rows of a later chunk are read.
int rank_rows(LeniaMlp* n, const float* x, uint32_t count, float* probs) {
    if (in_place(n, x)) {
        if (count > 0) touch_rows(x, (size_t)count * IN);
        // probabilities over their own rows leave by copy, after the launch has read them
        const bool apart = probs + (size_t)count * OUT <= x || x + (size_t)count * IN <= probs;
        if (count > 0 && apart && pageable_in_place(n->reads_host, probs, (size_t)count * OUT * 4)) {
            // no copy after the tiles: 1000 rows 30.5 -> 25.3 us, 19456 47.9 -> 36.0, 65536 74.0 -> 67.4
            touch_pages(probs, (size_t)count * OUT * 4, true);
            if (!rank(n, n->ps[0], x, count, probs)) return abandon(n, "mlp: launch failed");
        } else {
            for (uint64_t off = 0; off < count; off += DIRECT_ROWS) {
                const uint32_t B = count - off < DIRECT_ROWS ? (uint32_t)(count - off) : DIRECT_ROWS;
                if (!rank(n, n->ps[0], x + off * IN, B, n->pp)) return abandon(n, "mlp: launch failed");
                if (cudaMemcpyAsync(probs + off * OUT, n->pp, (size_t)B * OUT * 4, cudaMemcpyDeviceToHost, n->ps[0]) !=
                    cudaSuccess)
                    return abandon(n, "mlp: download failed");
            }
        }
        if (cudaStreamSynchronize(n->ps[0]) != cudaSuccess) return abandon(n, "mlp: predict failed");
        return check_err(n);
    }
    // chunk c runs on stream c % 2; its results leave after the next chunk has been queued, so that a copy
    // to or from pageable memory, which blocks this thread, overlaps a chunk's tiles
    const uint32_t chunks = (uint32_t)(((uint64_t)count + HALF - 1) / HALF);
    auto rows = [&](uint32_t c) { return c + 1 < chunks ? HALF : count - c * HALF; };
    for (uint32_t c = 0; c <= chunks; c++) {
        if (c < chunks) {
            const int h = c & 1;
            float *px = n->px + (size_t)h * HALF * IN, *pp = n->pp + (size_t)h * HALF * OUT;
            if (cudaMemcpyAsync(px, x + (size_t)c * HALF * IN, (size_t)rows(c) * IN * 4, cudaMemcpyHostToDevice, n->ps[h]) !=
                cudaSuccess)
                return abandon(n, "mlp: upload failed");
            if (!rank(n, n->ps[h], px, rows(c), pp)) return abandon(n, "mlp: launch failed");
        }
        if (c > 0) {
            const uint32_t d = c - 1;
            if (cudaMemcpyAsync(probs + (size_t)d * HALF * OUT, n->pp + (size_t)(d & 1) * HALF * OUT, (size_t)rows(d) * OUT * 4,
                                cudaMemcpyDeviceToHost, n->ps[d & 1]) != cudaSuccess)
                return abandon(n, "mlp: download failed");
        }
    }
    if (cudaStreamSynchronize(n->ps[0]) != cudaSuccess || cudaStreamSynchronize(n->ps[1]) != cudaSuccess)
        return abandon(n, "mlp: predict failed");
    return check_err(n);
}

}  // namespace

extern "C" {

LENIA_API int lenia_mlp_create(uint32_t seed, uint32_t max_batch, LeniaMlp** out) {
    if (!out || max_batch < 1 || max_batch > (1u << 22)) {
        set_thread_error("mlp: need an output pointer and 1 <= max_batch <= 4M");
        return LENIA_EINVAL;
    }
    *out = nullptr;
    LeniaMlp* n = new LeniaMlp();
    n->max_batch = (int)max_batch;
    const size_t B = max_batch;
    int dev = 0;
    bool ok = cudaGetDevice(&dev) == cudaSuccess &&
              cudaDeviceGetAttribute(&n->sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
              cudaDeviceGetAttribute(&n->reads_host, cudaDevAttrPageableMemoryAccessUsesHostPageTables, dev) == cudaSuccess &&
              cudaFuncSetAttribute(mlp_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM) == cudaSuccess &&
              cudaFuncSetAttribute(mlp_rank, cudaFuncAttributeMaxDynamicSharedMemorySize, RANK_SMEM) == cudaSuccess &&
              cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&n->ps[0], cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&n->ps[1], cudaStreamNonBlocking) == cudaSuccess && mal(n, &n->w, NPARAM) &&
              mal(n, &n->g, NPARAM) && mal(n, &n->m, NPARAM) && mal(n, &n->v, NPARAM) && mal(n, &n->wb, NPARAM) &&
              mal(n, &n->x, B * IN) && mal(n, &n->y, B * OUT) &&
              cudaHostAlloc((void**)&n->err, (B + 4) * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess &&
              mal(n, &n->px, (size_t)PREDICT_ROWS * IN) && mal(n, &n->pp, (size_t)DIRECT_ROWS * OUT);
    if (!ok) {
        lenia_mlp_destroy(n);
        set_thread_error("mlp: device allocation failed");
        return LENIA_ENOMEM;
    }
    *n->err = 0;
    n->loss = reinterpret_cast<float*>(n->err + 4);
    // He-uniform initialisation from the PCG hash, biases zero
    std::vector<float> w(NPARAM, 0.f);
    auto pcg = [](uint32_t v) {
        uint32_t s = v * 747796405u + 2891336453u;
        uint32_t x = ((s >> ((s >> 28u) + 4u)) ^ s) * 277803737u;
        return (x >> 22u) ^ x;
    };
    auto init = [&](int off, int count, int fan_in) {
        const float a = std::sqrt(6.0f / fan_in);
        for (int i = 0; i < count; i++) {
            const uint32_t r = pcg(pcg(pcg((uint32_t)(off + i)) ^ seed) ^ 0x9E3779B9u);
            w[off + i] = a * (2.0f * ((float)r * (1.0f / 4294967296.0f)) - 1.0f);
        }
    };
    init(P_W1, HID * IN, IN);
    init(P_W2, HID * HID, HID);
    init(P_W3, OUT * HID, HID);
    int rc = lenia_mlp_set_params(n, w.data(), w.size());
    if (rc) {
        lenia_mlp_destroy(n);
        return rc;
    }
    cudaMemsetAsync(n->m, 0, NPARAM * 4, n->stream);
    cudaMemsetAsync(n->v, 0, NPARAM * 4, n->stream);
    if (cudaStreamSynchronize(n->stream) != cudaSuccess) {
        lenia_mlp_destroy(n);
        return err("mlp: initialisation failed");
    }
    *out = n;
    return 0;
}

LENIA_API int lenia_mlp_destroy(LeniaMlp* n) {
    if (!n) return 0;
    for (cudaStream_t s : {n->stream, n->ps[0], n->ps[1]})
        if (s) cudaStreamSynchronize(s);
    for (void* p : n->allocs) cudaFree(p);
    if (n->err) cudaFreeHost(n->err);
    for (cudaStream_t s : {n->stream, n->ps[0], n->ps[1]})
        if (s) cudaStreamDestroy(s);
    delete n;
    return 0;
}

LENIA_API int lenia_mlp_param_count(uint32_t* count) {
    if (!count) return LENIA_EINVAL;
    *count = NPARAM;
    return 0;
}

LENIA_API int lenia_mlp_set_params(LeniaMlp* n, const float* host, size_t count) {
    if (!n || !host || count != (size_t)NPARAM) {
        set_thread_error("mlp: parameter vector has the wrong length");
        return LENIA_EINVAL;
    }
    if (cudaMemcpyAsync(n->w, host, NPARAM * 4, cudaMemcpyHostToDevice, n->stream) != cudaSuccess)
        return abandon(n, "mlp: upload failed");
    if (!each_param(n, to_bf16, n->w, n->wb, NPARAM)) return abandon(n, "mlp: launch failed");
    n->t = 0;
    return cudaStreamSynchronize(n->stream) == cudaSuccess ? 0 : err("mlp: set_params failed");
}

LENIA_API int lenia_mlp_get_params(LeniaMlp* n, float* host, size_t count) {
    if (!n || !host || count != (size_t)NPARAM) {
        set_thread_error("mlp: parameter vector has the wrong length");
        return LENIA_EINVAL;
    }
    if (cudaMemcpyAsync(host, n->w, NPARAM * 4, cudaMemcpyDeviceToHost, n->stream) != cudaSuccess ||
        cudaStreamSynchronize(n->stream) != cudaSuccess)
        return abandon(n, "mlp: download failed");
    return 0;
}

LENIA_API int lenia_mlp_gradients(LeniaMlp* n, const float* x, const float* y, uint32_t batch, float* grads,
                                  float* loss) {
    if (!n || !x || !y || !grads || batch < 1 || batch > (uint32_t)n->max_batch) {
        set_thread_error("mlp: bad batch");
        return LENIA_EINVAL;
    }
    if (int rc = batch_gradients(n, x, y, batch)) return rc;
    // straight into the caller's memory where kernels reach it: 1000 rows 65.3 -> 62.7 us against the driver's copy, which
    // waits for a change of engine
    if (pageable_in_place(n->reads_host, grads, NPARAM * 4)) {
        touch_pages(grads, NPARAM * 4, true);  // beside the tiles
        if (!each_param(n, copy_out, n->g, grads, NPARAM)) return abandon(n, "mlp: launch failed");
    } else if (cudaMemcpyAsync(grads, n->g, NPARAM * 4, cudaMemcpyDeviceToHost, n->stream) != cudaSuccess) {
        return abandon(n, "mlp: download failed");
    }
    return mean_loss(n, batch, loss);
}

LENIA_API int lenia_mlp_train_step(LeniaMlp* n, const float* x, const float* y, uint32_t batch, float lr, float* loss) {
    if (!n || !x || !y || batch < 1 || batch > (uint32_t)n->max_batch || !(lr > 0.f)) {
        set_thread_error("mlp: bad batch or learning rate");
        return LENIA_EINVAL;
    }
    if (int rc = batch_gradients(n, x, y, batch)) return rc;
    n->t++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)n->t), c2 = 1.f - std::pow(b2, (float)n->t);
    if (!each_param(n, adam, n->w, n->g, n->m, n->v, n->wb, NPARAM, lr, b1, b2, 1e-8f, c1, c2))
        return abandon(n, "mlp: launch failed");
    return mean_loss(n, batch, loss);
}

LENIA_API int lenia_mlp_predict(LeniaMlp* n, const float* x, uint32_t count, float* probs) {
    if (!n || !x || !probs) {
        set_thread_error("mlp: NULL argument");
        return LENIA_EINVAL;
    }
    // Over their own rows, behind the start (12 bytes a row never catch up with 64), the first chunk's probabilities could
    // lie where later rows are yet to be read: they wait in a buffer.
    if (count > HALF && probs > x && probs < x + (size_t)count * IN) {
        const size_t bytes = (size_t)count * OUT * sizeof(float);
        float* all = static_cast<float*>(malloc(bytes));
        if (!all) {
            set_thread_error("mlp: no host memory for probabilities over their own rows");
            return LENIA_ENOMEM;
        }
        const int rc = rank_rows(n, x, count, all);
        if (!rc) memcpy(probs, all, bytes);
        free(all);
        return rc;
    }
    return rank_rows(n, x, count, probs);
}

}  // extern "C"
