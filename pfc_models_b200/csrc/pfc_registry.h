// Kernel lookup across translation units. The step kernels are instantiated in
// several .cu files (one per precision and variant) that compile in parallel; the
// plan code finds them through these functions.
#pragma once
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "pfc_extv.h"

namespace pfc {

// Radix-set codes of the run-time kernels: kRadixPow2, kRadixSmall and kRadixAll
// (pfc_fft.cuh) select the two-buffer kernels (pfc_mixed.cuh); the codes below the one-buffer
// kernels (pfc_kernels.cuh, 1024-thread blocks) for transforms whose two buffers exceed
// kMixedSmem of shared memory (FP64 8192 points), with power-of-two radices or with the
// radices up to 7. (Lengths with a factor 11 or 13 always fit two buffers.)
constexpr int kRadixPow2Big = 2;
constexpr int kRadixSmallBig = 6;
constexpr size_t kMixedSmem = 200 * 1024;
// most threads of a Parseval or export CTA, which hold one column of 4096 points or more
constexpr int kParThreads = 512;

// log2 sizes of the power-of-two step kernels: row transforms of M = nx/2 points,
// column transforms of ny points
constexpr int kFastMinLog = 5, kFastMaxLogRow = 12, kFastMaxLogCol = 13;

// Work-queue step kernel of one precision (pfc_queue.cuh; pfc_queue_f32.cu, pfc_queue_f64.cu).
template <class T>
struct QueueInst {
  static void* kernel();
};

struct FastKernel {
  void* fn = nullptr;  // kernel entry, for cudaLaunchKernel
  int tpf = 0;         // threads per transform
};

// Power-of-two step kernels with EE complex values per thread (pfc_fast.cuh).
template <class T, int EE>
struct FastInst {
  static bool row(int lg, int model, FastKernel* out);
  static bool col(int lg, FastKernel* out);
  // appends the pass tables of sequences A and B of a 2^lg-point transform
  static bool tables(int lg, std::vector<long double>& tw, int& offA, int& offB);
};

// Power-of-two row step kernels with paired butterflies (pfc_rowpair.cuh) of 2^lg-point rows,
// lg >= kPairMinLog (a tile of 32-point rows is less than a warp): values per thread, and rows
// per CTA for a variant of `tile` rows (0: none asked for), by length, precision and model.
// Rows of up to 512 points take 8 values a thread (the most threads; us per step on B200 with 8
// / 16 values: 256^2 FP64 6.7 / 6.8, FP32 6.8 / 7.3, 512^2 8.0 / 8.5 and 7.4 / 8.7, 1024^2 log
// 20.6 / 21.1 and 13.6 / 16.2), longer ones as many as 128 registers hold (2048^2 FP64 8 / 16
// values 56.9 / 51.7, FP32 16 / 32 values 31.2 / 30.2, 8192^2 598 / 580). Tiles hold 64-byte
// runs where a CTA of them fits an SM, and in FP32 32-byte ones for single plans of 256- and
// 512-point rows, whose CTAs are few (512^2 7.4 against 7.7, 1024^2 log 13.6 against 14.2; a
// batch of 24 512^2 plans prefers 8 rows, 41.3 against 43.1 us) and for 2048 points (121 against
// 124). The log model's logarithms, inlined per value, make the widest kernel's code long: 16
// values for 1024 and 2048 points (2048^2 FP32 35.1 against 36.5, 4096^2 137 against 165; 8192^2
// 690 against 687), and FP64 tiles of 2 rows at 2048 points (275 against 286). One-lane kernel
// at its tuned variants: 256^2 FP64 8.1, FP32 8.2; 512^2 9.2, 8.5; 2048^2 59.3, 32.9; 4096^2
// 260, 138 (packed, TMA); 8192^2 1375, 615 (packed, TMA); log 1024^2 22.5, 14.8, 2048^2 70.7,
// 42.5, 4096^2 300, 174, 8192^2 FP32 780.
constexpr int kPairMinLog = 6;
constexpr int pair_ee(bool fp64, int lg, bool log) { return lg <= 9 ? 8 : fp64 || (log && lg <= 11) ? 16 : 32; }
constexpr int pair_rows(bool fp64, int lg, bool log, int tile) {
  if (fp64) return lg <= (log ? 10 : 11) ? 4 : 2;
  return lg == 10 || (lg <= 9 && (tile >= 8 || (!tile && lg <= 7))) ? 8 : 4;
}

struct PairKernel {
  void* fn = nullptr;
  int threads = 0;
  size_t smem = 0;
  std::vector<int> radices;   // of sequence A
};
template <class T>
struct PairInst {
  static bool row(int lg, int rows, int model, PairKernel* out);
};

// Register-resident step kernels for transforms of N = ODD * 2^k points, ODD = 3, 5, 7
// and k = kMixMinLog2 .. kMixMaxLog2 (pfc_fastmix_inst.cuh), by transform length.
constexpr int kMixMinLog2 = 4, kMixMaxLog2 = 9;
template <class T>
struct MixInst {
  static bool row(int n, int model, FastKernel* out);
  static bool col(int n, FastKernel* out);
  static bool tables(int n, std::vector<long double>& tw, int& offA, int& offB);
  static int values_per_thread(int n);
};

// Two-lane packed FP32 step kernels (pfc_pack_step.cuh), `ee` = 8 or 16 complex values
// per lane and thread: row transforms of 2^lg points (M = nx/2), column transforms of
// 2^lg points (ny). Their pass tables are float4 entries (c, c, s, s), appended to `tw`
// as two complex slots each, at even (16-byte aligned) offsets; pack_real_table appends
// the real-packing table exp(-2 pi i k / nx), k < nx/2, in the same form.
constexpr int kPackMinLog = 6, kPackMaxLogRow = 12, kPackMaxLogCol = 13;
bool pack_row(int lg, int ee, int model, FastKernel* out);
bool pack_col(int lg, int ee, FastKernel* out);
bool pack_tables(int lg, int ee, std::vector<long double>& tw, int& offA, int& offB);
void pack_real_table(int nx, std::vector<long double>& tw, int& off);

// Mixed-radix kernels (pfc_kernels.cuh), by mode (kRow* / kCol*) and radix set.
template <class T>
struct GenericInst {
  static void* row(int mode, int model, int rset);
  static void* col(int mode, int rset);
};

// Mode entries of the 3-mode diagnostics (pfc_diag.cu), built on the host from the
// reference's k-vector sets: the list (with repeats) whose |n_hat| each set averages,
// and the distinct entries of the rebuilt spectrum with their half-spectrum weights
// (set -1: the DC entry, which keeps n_hat(0, 0)). Indices are flat in the
// (ny, nx / 2 + 1) half spectrum.
constexpr int kDiagMaxModes = 64;
struct DiagModes {
  double sign;
  int n_list, n_uniq;
  int list_flat[kDiagMaxModes], list_set[kDiagMaxModes];
  int uniq_flat[kDiagMaxModes + 1], uniq_set[kDiagMaxModes + 1];
  double uniq_w[kDiagMaxModes + 1];
};
cudaError_t launch_diagnose_modes(const double* field, const double* spec, int nx, int ny, const DiagModes& m,
                                  double* partials, double* out6, cudaStream_t stream);
cudaError_t launch_frozen_moments(const double* field, const double* spec, int nx, int ny, double fx, double fy,
                                  double temp, double g, double v0, double* partials, double* out4,
                                  cudaStream_t stream);
cudaError_t launch_defect_screen(const double* field, const double* spec, int nx, int ny, double fx, double fy,
                                 double* partials, double* out4, cudaStream_t stream);
int diagnose_partials_needed();

// Whole-grid step kernel for small FP64 mixed-radix grids (pfc_onecta.cuh): one CTA per
// plan runs nsteps steps with the grid in shared memory; `table` holds the plans'
// buffers (BatchBufs) at the starting parity, `count` entries.
template <class T> struct RowArgs;
template <class T> struct ColArgs;
struct BatchBufs;
constexpr int kOneCtaMaxThreads = 256;
constexpr size_t kOneCtaMaxSmem = 96 * 1024;   // two CTAs per SM
size_t onecta_smem_bytes(int m, int ny, int row_ld, int col_ld);
// raises the dynamic shared memory limit of a model's and radix set's kernels
cudaError_t onecta_allow_smem(size_t bytes, int model, int rset);
// the kernel at one CTA an SM, or (dense) at two
template <int MODEL, int RSET> struct OnectaInst { static void* kernel(bool dense); };
bool onecta_supported(int rset);
cudaError_t launch_onecta_step(const RowArgs<double>& ra, const ColArgs<double>& ca, const BatchBufs* table,
                               int count, long long nsteps, int model, int rset, bool dense, int threads,
                               size_t smem, cudaStream_t stream);

// The same step with dense transforms on the FP64 tensor cores (pfc_dense.cu).
struct DenseArgs {
  int m, ny, nyh;                  // half row length, column length, coefficients a column
  int tr, kr, tc, kc;              // 8-wide output tiles and 4-deep steps of the row and column matrices
  int ys, ks, cpad;                // strides of the [.][y] and [.][ky] arrays, real columns padded to 8
  int size_a, size_b;              // doubles of the two work areas
  const double2 *row_tab, *col_tab;
  double g, min_phi, min_log, scale;
  int clamp;
};
size_t dense_shape(int m, int ny, DenseArgs& a);           // fills the sizes; bytes of shared memory
int dense_products(const DenseArgs& a);                    // m8n8k4 products of a step
// Plans of up to this many products a step take the dense transforms. Their cost grows with
// the square of the sides. B200, us a step, one cell / 296 cells in one batch, dense against
// FFT passes: 28 x 24 (224 products) 2.0 / 2.8 against 6.0 / 6.3, 48 x 20 (512) 3.7 / 4.8
// against 5.5 / 6.2, 30 x 50 (672) 4.2 / 5.9 against 6.4 / 7.6, 32 x 56 (932) 5.4 / 7.9
// against 6.6 / 7.8 and for the log model 7.4 / 10.6 against 8.0 / 9.6 (dense before it took the mean
// out of its transforms, 0.13 us a step more on 28 x 24).
constexpr int kDenseMaxProducts = 800;
// appends the (w cos, w sin) fragments of length n; root = exp(-2 pi i k / n), k < n
void dense_table(int n, const std::vector<long double>& root, std::vector<long double>& tw);
cudaError_t dense_allow_smem(size_t bytes);
cudaError_t launch_dense_step(const DenseArgs& args, const BatchBufs* table, int count, long long nsteps, int model,
                              size_t smem, cudaStream_t stream);

// Log PFC with an external potential (pfc_extv.cu): the decision and the rebuild as kernels of
// their own, for plans whose row or column pass runs the one-buffer kernels.
cudaError_t launch_extv_decide(const double* minmax, int nparts, ExtvState* st, double g, cudaStream_t s);
cudaError_t launch_extv_coef(const ExtvCoefArgs& a, const ExtvState* st, cudaStream_t s);

// Vacancy location on a local density field (pfc_track.cu), count > 0.
cudaError_t launch_locate_vacancies(const double* field, int nx, int ny, double dx, double dy, double* xy,
                                    int count, int32_t* status, cudaStream_t stream);

}  // namespace pfc
