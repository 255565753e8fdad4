// bk_internal.h -- declarations shared by the translation units of the
// library (not part of the C ABI).
#pragma once

#include <cuda_runtime.h>

#include "bk_gpu.h"

namespace bkg {

struct DevCtx;

constexpr int kMaxDevices = 64;

int current_device();          // cudaGetDevice, or -1

// BK5's built-in choice for BK_KERNEL_AUTO: the column kernel for the
// FP32-storage engines (2: FP32, 3: mixed) with G in the column layout at
// p <= 3 and at p = 5 with the mass term, the sweep kernel otherwise.  Measured
// on GB300, mixed form, us sweep / column at 1 M, 4 M and 16 M points, with the
// mass term: p = 1 11.2 / 9.9, 35.3 / 31.7, 129 / 118; p = 2 11.6 / 10.6, 36.4 /
// 32.4, 124 / 120; p = 3 10.5 / 8.7, 30.1 / 25.3, 102 / 90; p = 4 11.0 / 10.8,
// 29.7 / 32.6, 101 / 117; p = 5 11.2 / 10.4, 31.8 / 31.5, 107 / 112; p = 6 11.3 /
// 11.2, 32.3 / 34.6, 105 / 126.  Without it: p = 2 10.8 / 10.3, 33.2 / 31.5, 116 /
// 117; p = 3 9.4 / 8.4, 26.2 / 23.6, 88 / 83; p = 4 10.3 / 10.5, 27.7 / 31.0, 92 /
// 113; p = 5 10.3 / 10.1, 28.3 / 30.3, 96 / 109.
inline int bk5_builtin_auto(int p, int eng, int layout, bool with_mass)
{
    return (eng >= 2 && layout == 2 && (p <= 3 || (p == 5 && with_mass))) ? BK_KERNEL_COLUMN : BK_KERNEL_SWEEP;
}
int sm_count();                // SMs of the current device
DevCtx dev_ctx();              // status word and wait limit of the current device

#define BK_DECLARE_ENGINE(sfx)                                                                                    \
    int launch_bk5_##sfx(int p, long long E, const double* D, const void* G, const void* u, const void* mass,    \
                         double lambda, void* v, int F, int layout, int eb, int kernel, int gform, cudaStream_t s); \
    int launch_bk1_##sfx(int p, long long E, const double* B, const void* jxw, const void* u, void* v, int eb,   \
                         int jxw_t, cudaStream_t s);                                                             \
    int launch_bk3_##sfx(int p, long long E, const double* B, const double* D, const void* G, const void* k,     \
                         const void* u, void* v, int eb, int gform, cudaStream_t s);                                        \
    int bk5_sweep_##sfx##_L0(int p, int F, const double* D, long long E, const void* u, const void* G,  \
                             const void* mass, double lambda, void* v, int gform, cudaStream_t s);                          \
    int bk5_sweep_##sfx##_L1(int p, int F, const double* D, long long E, const void* u, const void* G,  \
                             const void* mass, double lambda, void* v, int gform, cudaStream_t s);                          \
    int bk5_sweep_##sfx##_L2(int p, int F, const double* D, long long E, const void* u, const void* G,  \
                             const void* mass, double lambda, void* v, int gform, cudaStream_t s);                               \
    int bk5_col_##sfx##_L0(int p, int F, int eb, const double* D, long long E, const void* u, const void* G,    \
                           const void* mass, double lambda, void* v, cudaStream_t s);                            \
    int bk5_col_##sfx##_L1(int p, int F, int eb, const double* D, long long E, const void* u, const void* G,    \
                           const void* mass, double lambda, void* v, cudaStream_t s);                            \
    int launch_bk3_adjoint_##sfx(int p, long long E, const double* B, const double* D, const void* G,           \
                                 const void* k, const void* u, const void* res, void* dk, void* dG,              \
                                 int gform, cudaStream_t s);                                                                \
    int bk5_col_##sfx##_L2(int p, int F, int eb, const double* D, long long E, const void* u, const void* G,    \
                           const void* mass, double lambda, void* v, cudaStream_t s);

BK_DECLARE_ENGINE(dfma)
BK_DECLARE_ENGINE(ff)
BK_DECLARE_ENGINE(f32)
BK_DECLARE_ENGINE(mixed)

}  // namespace bkg
