// Internal declarations shared by the engine's translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/lenia_gb300.h"

namespace lenia {

// One kernel's per-step parameters on the device.
struct DevKernel {
    int src, dst;
    float mu, sigma, weight;
};

// One world on the device.  Layouts (HBM):
//   state [C][H][W] float                               channel-major, row-major (reference layout)
//   spec  [C][W/(2*TC)][H][TC] float2   half-spectrum along x of every row, in tiles of TC
//                                 columns so that a column pass reads one contiguous block;
//                                 column 0 packs the DC column (real part) with the Nyquist
//                                 column W/2 (imaginary part)
//   conv  [K][W/(2*TC)][H][TC] float2   per-kernel convolved spectrum (aliases spec when C = K = 1)
//   khat  [K][W/2+1][HQ] float    real, even kernel spectrum for ky in [0, H/2], times 1/(W*H);
//                                 HQ = khat_stride(H) >= H/2+1
struct DevWorld {
    int W, H, C, K, rule;
    float dt;
    int HQ;
    float* state;
    float2* spec;
    float2* conv;
    const float* khat;
    float* u_out;  // U_k fields [K][H][W] when a row pass runs in MODE_U
    DevKernel kern[LENIA_MAX_KERNELS];
};

// Spectrum columns per tile: a column pass CTA transforms TC columns of length H.
constexpr int TC = 2;

// Work items.
// A column item: spectrum tile `tile` of channel `chan` with kernel `kernel` (FP32 pass); the
// tensor-core groups use world, chan and the first tile of the group.
struct ColItem { int world, chan, tile, kernel; };
// A row item: rows row0.. of one world.  For Lenia worlds one item per target channel `chan`
// (its kernels, its state update and its forward transform); other rules use chan = 0 and every
// channel.
struct RowItem { int world, row0, chan, pad; };

enum RowMode { MODE_STEP = 0, MODE_FORWARD = 1, MODE_U = 2 };

// Where and how a pass is launched.
// overlap: a programmatic dependent launch, whose CTAs may start before the kernel ahead of it on the
// stream has finished; only for a launch that directly follows another FP32 pass on the same
// stream (every pass waits for the kernel ahead of it, griddepcontrol.wait, before it touches what that
// kernel reads or writes).  A CTA's set-up (its item, the world, stage tables, the kernel spectrum's
// columns) then runs before that wait: 0.5 us a launch at every size, 1024 x 1024 alone 11.95 -> 11.1 us
// a generation.
// early: the pass lets the launch after it start before its own last stage or its spectrum stores, not
// only as its CTAs end.
struct LaunchOn {
    cudaStream_t s;
    bool overlap, early;
    LaunchOn(cudaStream_t stream, bool overlap_ = false, bool early_ = false) : s(stream), overlap(overlap_), early(early_) {}
};
template <class... P, class... A>
bool launch_pass(void (*kernel)(P...), int grid, int threads, size_t smem, LaunchOn on, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = on.s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = on.overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess;
}

// Fused FP32 path (step_fp32_*.cu).  Every size is built in two launch variants: variant 0 caps registers
// at 64 or 80 per thread (more resident CTAs), variant 1 at 128 (and gives a row item from 768 wide up
// two CTAs, see row_cta_seqs).  The column pass has two more: variant 2, the paired build (both columns of a tile
// in one sequence of f32x2 pairs, half the threads), and variant 3 (COL_VARIANTS).  The row
// launcher picks its general build from its `general` argument.  Launchers return false if the
// size is not built.
bool launch_col_fp32(int H, int variant, const DevWorld* worlds, const ColItem* items, int nitems,
                     const float2* tw, LaunchOn s);
bool launch_row_fp32(int W, int variant, int mode, int general, const DevWorld* worlds, const RowItem* items,
                     int nitems, const float2* tw, LaunchOn s);
size_t col_smem_bytes(int H);
size_t row_smem_bytes(int W, int general);
// Column-pass launch variants (launch_col_fp32): 0, 1 scalar builds at two register caps, 2 the paired
// build, 3 the scalar radix-16 build (1024) or the scalar build with one column a CTA (2048 and more)
constexpr int COL_VARIANTS = 4;
// whether variant 3 is a build of its own at height H
bool col_has_variant3(int H);
// whether the scalar column pass of height H holds 24 or 32 elements a thread (radix-32 plans, the
// larger two-stage transforms)
bool col_wide(int H);
int row_item_rows(int W, int general);  // rows per row-pass item: 2, 4 or 8 (row_seqs)
int max_smem_optin();

// Cluster-resident step (resident.cu): one launch advances every world of a square size class of
// side N (128, 192, 256, 384 or 512; one channel, one Lenia kernel) `gens` generations, one
// thread-block cluster of N/32 CTAs per world.  world_ids: the class's world indices (device).
// err: a device int set to 1 if a cluster sync gave up.  A zero-world call only configures the
// kernel (outside any stream capture).
// Each size is built in RESIDENT_VARIANTS launch variants (sequences per batch, register budget).
constexpr int RESIDENT_VARIANTS = 3;
bool resident_supported(int N);
// co-resident clusters of a variant on this GPU (0: the launch cannot run); configures the kernel
int resident_clusters_that_fit(int N, int variant);
bool launch_resident(int N, int variant, const DevWorld* worlds, const int* world_ids, int nworlds, int gens,
                     const float2* tw, int* err, cudaStream_t s);

// Persistent step (persist.cu): one launch advances every world of a square, one-channel, one-kernel
// Lenia size class of side N through `gens` generations, with the two-pass step's column and row
// items (cols: nc a world, rows: nr a world, world after world) claimed in order by a grid of
// resident CTAs.  ctl: persist_ctl_words(nworlds) ints, zeroed before every launch.  err: two device
// ints, [0] set to 1 if a wait gave up, [1] the waits' poll limit + 1 (0: the default; 1: every
// dependency wait gives up at once, a test hook).  capacity (optional): CTAs the GPU holds at once.
// A zero-world call only configures the kernel (outside any stream capture).
// variant: 0 at most 64 registers a thread, 1 at most 128 (as the two-pass step's launch variants).
constexpr int PERSIST_VARIANTS = 2;
bool persist_supported(int N);
int persist_ctl_words(int nworlds);
bool launch_persist(int N, int variant, const DevWorld* worlds, const ColItem* cols, const RowItem* rows, int nworlds,
                    int ncol, int nrow, int gens, const float2* tw, int* ctl, int* err, cudaStream_t s,
                    int* capacity = nullptr);

// Seeding and statistics (seed.cu).
void launch_seed_patches(float* state, int W, int H, uint32_t seed, const int4* patches, int npatch,
                         cudaStream_t s);
void launch_seed_tiles(float* state, int W, int H, uint32_t seed, const float* pattern, int pw, int ph,
                       int spacing, cudaStream_t s);
// Whether kernels take a range of the caller's memory where it is: pageable memory that the GPU reaches through the host's page
// tables (reads_host: cudaDevAttrPageableMemoryAccessUsesHostPageTables), 16-byte aligned, of at most 1 MiB.  Above, the
// driver's copies reach the link's rate as well, and pages that are not there yet cost more from the GPU (64 MiB into
// fresh pages 3.7 -> 21.5 ms).
bool pageable_in_place(int reads_host, const void* p, size_t bytes);
// Touches every page of such a range from the host first: pages not there yet get their place from the host, and a bad
// range faults there, not on the GPU.
void touch_pages(void* p, size_t bytes, bool write);
// count floats, a multiple of 4, between 16-byte aligned places; whether this launch succeeded
bool launch_copy_words(float* dst, const float* src, size_t count, cudaStream_t s);
// max_sides: the largest W + H of the worlds
bool launch_world_stats(const DevWorld* worlds, int nworlds, int max_sides, float* out, cudaStream_t s);
void launch_seed_rule(float* state, int W, int H, uint32_t seed, int kind, cudaStream_t s);
void launch_render(const float* state, int W, int H, float ox, float oy, float scale, int n, int out_w, int out_h,
                   int palette, uchar4* out, cudaStream_t s);

// The message lenia_last_error(NULL) returns on this thread (calls that have no context).
void set_thread_error(const std::string& msg);

// Tile-layout helpers on the host.
inline size_t spec_elems(int W, int H) { return (size_t)(W / 2) * H; }
inline int spec_tiles(int W) { return W / (2 * TC); }
// Row stride of the kernel spectrum (floats): H/2+1 rounded up to a multiple of 4, so that
// every row starts 16-byte aligned and can be moved by a bulk copy.
inline int khat_stride(int H) { return (H / 2 + 1 + 3) / 4 * 4; }

}  // namespace lenia
