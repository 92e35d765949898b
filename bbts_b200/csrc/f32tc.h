// FP32 products on the tensor cores (gemm_f32tc.cuh): host side. An operand is
// described by the gather that lays it out as [batch][rows][pitch]; its three
// bf16 planes and the maxima of its chunks live in caller-provided workspace.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>
#include <cuda_runtime_api.h>
#include "contraction.h"

namespace bbx {

// One operand: `batch` matrices of rows x cols, in planes of pitch `pitch`.
// K-major (mn false): rows are the M or N dimension and cols K; mn: the reverse.
struct F3Mat {
  const float* src = nullptr;
  GatherArgs g{};
  bool mn = false;
  bool split = true;           // false: another operand of the group with the same ws is split, of the same layout
  long long rows = 0, cols = 0, pitch = 0, batch = 1;
  void* ws = nullptr;  // f3_mat_bytes, 256-byte aligned
};

// C = alpha op(A) op(B) (+ beta C) (+ bias), batched. a, b: indices of the operands.
struct F3Spec {
  int a = 0, b = 0;
  float* c = nullptr;
  const float* bias = nullptr;
  int m = 0, n = 0, k = 0;
  long long ldc = 0, c_batch = 0;
  bool c_col = false;
  float alpha = 1.f, beta = 0.f;
};

// True when an m x n x k product (each of `batch`) runs on the tensor cores
// rather than on the SIMT kernels. The per-call and the grouped paths share
// this rule and give the same bits, except where there is no room for the planes
// (per call: no scratch; a compiled list: built without them), and for a dense
// product under stream capture: those run the SIMT kernels.
bool f3_wanted(long long m, long long n, long long k, long long batch);

// While one lives (with on = true), the f32 products that its thread enqueues keep the SIMT
// kernels' single FMA chain. The executors use it for products whose result
// reaches a ReLU (directly or through adds): the sign of a pre-activation near 0
// decides its mask, and a flipped mask moves a whole term of a gradient (1e-3 of its
// norm from one flip in 10^6), so these masks stay those of the plain FP32 path, bit for bit.
// Other ops between the product and the ReLU, and a ReLU in a later list, are not followed.
class FmaChain {
 public:
  explicit FmaChain(bool on);
  ~FmaChain();
  FmaChain(const FmaChain&) = delete;
  FmaChain& operator=(const FmaChain&) = delete;
  static bool active();

 private:
  bool before_;
};

// The same for a contraction (lowered for the tensor cores). The SIMT kernel's
// grid limits hold here too.
bool f3_contraction_wanted(const ContractionLowering& L);

// A row-major rows x cols matrix of pitch ld (elements), `batch` of them `stride` apart.
F3Mat f3_dense(const float* src, long long rows, long long cols, long long ld, long long batch, long long stride, bool mn);
// The operands and the product of a contraction lowered for the tensor cores; C is the staged or direct output.
void f3_contraction(const ContractionLowering& L, const float* lhs, const float* rhs, float* c, float alpha, F3Mat* lc,
                    F3Mat* rc, F3Spec* out);
size_t f3_mat_bytes(const F3Mat& m);

// Enqueues the split and the product of one spec (mats[spec.a], mats[spec.b]).
int f3_run(const F3Mat* mats, const F3Spec& spec, void* stream);

// A group: every operand split by one launch, every product in one launch (per
// 256 products). Tables live on the device until destroyed.
struct F3Plan;
int f3_plan_create(const F3Mat* mats, int n_mats, const F3Spec* specs, int n_specs, F3Plan** out);
int f3_plan_launch(F3Plan* p, void* stream);
void f3_plan_destroy(F3Plan* p);
int f3_init();  // shared-memory opt-in, once per device, outside any capture

// A group of products on the SIMT kernels, one launch per operand layout.
struct F32SimtSpec {
  const float *a, *b;
  float* c;
  int m, n, k, trans_a, trans_b;
  long long lda, ldb, ldc;
};
struct F32SimtPlan;
int f32_simt_plan_create(const F32SimtSpec* specs, int n, F32SimtPlan** out);
int f32_simt_plan_launch(F32SimtPlan* p, void* stream);
void f32_simt_plan_destroy(F32SimtPlan* p);

// Stream-ordered scratch from the library's pool (per device). The pool keeps
// at most kScratchKeep bytes across synchronisations. nullptr when the device is
// out of memory; with `must`, only after scratch_reclaim.
void* scratch_alloc(size_t bytes, void* stream, bool must = false);
bool capturing(cudaStream_t st);
void scratch_free(void* p, void* stream);
// Gives back what the pool holds and nothing uses; reclaim first waits for the device, so
// that blocks whose release is still queued are among it. Before any allocation of the library's is
// reported as failed; not by a thread that captures a stream.
void scratch_trim();
void scratch_reclaim();

// cudaMalloc, once more after scratch_reclaim when the device is out of memory; what still fails
// counts in failed_allocs (of the calling thread). No error stays behind for a launch check.
cudaError_t device_alloc(void** p, size_t bytes);
unsigned& failed_allocs();

// 3-D bf16 tensor map: dims (cols, rows, planes), 128-byte swizzle (abi_kernels.cu).
int make_map3(void* map, const void* base, long long cols, long long rows, long long z, long long pitch,
              long long z_stride, int box_cols, int box_rows);

}  // namespace bbx
