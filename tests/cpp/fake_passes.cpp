// Stand-ins for the passes of the engine (step_fp32*.cu, step_tc*.cu, resident.cu, persist.cu, step_radix2.cu), for tests of the
// context's host code over fake_cudart.cpp: every launch succeeds and does nothing; sizes and item shapes are those of a
// plain build.
#include "../../auto_gb300/csrc/step_radix2.cuh"
#include "../../auto_gb300/csrc/step_tc.cuh"

namespace lenia {

bool launch_col_fp32(int, int, const DevWorld*, const ColItem*, int, const float2*, LaunchOn) { return true; }
bool launch_row_fp32(int, int, int, int, const DevWorld*, const RowItem*, int, const float2*, LaunchOn) { return true; }
size_t col_smem_bytes(int) { return 1 << 10; }
size_t row_smem_bytes(int, int) { return 1 << 10; }
bool col_has_variant3(int) { return false; }
bool col_wide(int) { return false; }
int row_item_rows(int, int) { return 2; }
int max_smem_optin() { return 227 << 10; }

bool resident_supported(int) { return false; }
int resident_clusters_that_fit(int, int) { return 0; }
bool launch_resident(int, int, const DevWorld*, const int*, int, int, const float2*, int*, cudaStream_t) { return true; }
bool persist_supported(int) { return false; }
int persist_ctl_words(int) { return 1; }
bool launch_persist(int, int, const DevWorld*, const ColItem*, const RowItem*, int, int, int, int, const float2*, int*, int*,
                    cudaStream_t, int*) {
    return true;
}

bool tc_supports(int) { return false; }
int tc_columns_per_group(int) { return 2; }
int tc_setup(TcPlan&, int, std::string*) { return 0; }
int tc_prepare_size(TcPlan&, int, int, std::string*) { return 0; }
bool launch_col_tc(const TcPlan&, int, int, int, const DevWorld*, const ColItem*, int, const float2*, cudaStream_t, int) { return true; }
int tc_check_error(TcPlan&, std::string*) { return 0; }
int tc_set_wait_limit(TcPlan&, int, std::string*) { return 0; }
void tc_release(TcPlan&) {}
bool tc_row_supports(int) { return false; }
int tc_row_group_rows(int) { return 4; }
int tc_row_prepare(TcPlan&, int, int, std::string*) { return 0; }
bool launch_row_tc(const TcPlan&, int, int, const DevWorld*, const RowItem*, int, int, const float2*, cudaStream_t) { return true; }
int tc_selftest(int, int, int, const float*, const float*, float*, std::string*) { return 0; }

void r2_enqueue_kernel_spectra(R2World&, const R2Shape*, const float*, cudaStream_t) {}
void r2_enqueue_convolve(R2World&, cudaStream_t) {}
void r2_enqueue_step(R2World&, cudaStream_t) {}

}  // namespace lenia
