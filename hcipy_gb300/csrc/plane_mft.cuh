// Tensor-core form of the plain-precision matrix Fourier transform (complex64 and complex128 plans); see
// plane_gemm.cuh for its arithmetic.
#pragma once

#include "hx_common.cuh"

namespace hx {

struct PlaneMft;

// Scratch below which hx_mft_execute refuses a call (mft.cu).  hx_mft_workspace_bytes may ask for more, with which
// the transform runs on the tensor cores; a caller that cannot give it gets the CUDA-core form.
size_t mft_least_workspace_bytes(const hx_mft_plan* p, int direction, int batch);

// Whether a transform between these grids may take the tensor-core form at all (a plan then keeps its operands).
bool plane_mft_fits(int nx, int ny, int nu, int nv, int dtype, bool weighted);
// Builds the cut phase matrices from device coordinate and weight arrays (weights may be NULL).  *out is NULL, without an
// error, where there is no memory for them.
int plane_mft_create(int dtype, int nx, int ny, int nu, int nv, const double* x, const double* y, const double* u,
                     const double* v, const double* wx, const double* wy, const double* wu, const double* wv,
                     cudaStream_t stream, PlaneMft** out);
void plane_mft_destroy(PlaneMft* p);
// Scratch of one call, 0 where the transform is left to the CUDA cores (see `takes` in plane_mft.cu).
size_t plane_mft_workspace_bytes(const PlaneMft* p, int direction, int batch);
// One transform; out, mask and src are of the plan's type.  throughput: no K split (other transforms run beside it).
int plane_mft_execute(const PlaneMft* p, int direction, int batch, const void* in, void* out, double are, double aim,
                      int epilogue, const void* mask, const void* src, bool throughput, void* ws, cudaStream_t stream);
// Status word of the bounded device waits (HX_OK or HX_ERR_TIMEOUT); synchronizes with the device.
int plane_mft_status(const PlaneMft* p, int reset);

}  // namespace hx
