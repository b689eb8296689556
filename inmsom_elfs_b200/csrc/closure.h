// Learned closure on the resident state of a context: the feature stencil,
// the fused inference + forcing update, and the per-point factors that turn
// a velocity tendency into the step's RHS units.
#pragma once

#include <cuda_runtime.h>

namespace inmsom {
namespace closure {

// launch on s with programmatic stream serialisation: the kernel's blocks may
// start while the stream's last kernel ends, and wait for it themselves
// (griddepcontrol.wait) before they read what it wrote
template <typename... P, typename... A>
cudaError_t launch_after(void (*k)(P...), int grid, int block, size_t smem, cudaStream_t s, A... a)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, P(a)...);
}

// the network's sizes and its parameter block (see closure.cu)
namespace net {
constexpr int KIN = 48, HID = 64, NOUT = 2, N3 = 8;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + KIN * HID, OFF_W2 = OFF_B1 + HID, OFF_B2 = OFF_W2 + HID * HID,
              OFF_W3 = OFF_B2 + HID, OFF_B3 = OFF_W3 + HID * N3, NPARAM = OFF_B3 + N3;
// A CTA's partial sums of the gradient hold dW1, dW2, dW3 column by column,
// each column with its bias gradient as the last row, then the loss
constexpr int ROWS1 = KIN + 1, ROWS2 = HID + 1;
constexpr int PART_W2 = HID * ROWS1, PART_W3 = PART_W2 + HID * ROWS2;
static_assert(PART_W3 + N3 * ROWS2 == NPARAM, "one partial sum per parameter");
// the parameter that partial sum i belongs to
__host__ __device__ constexpr int partial_param(int i)
{
    if (i < PART_W2) return i % ROWS1 < KIN ? OFF_W1 + i % ROWS1 * HID + i / ROWS1 : OFF_B1 + i / ROWS1;
    const bool last = i >= PART_W3;
    const int j = i - (last ? PART_W3 : PART_W2), row = j % ROWS2, col = j / ROWS2;
    if (last) return row < HID ? OFF_W3 + row * N3 + col : OFF_B3 + col;
    return row < HID ? OFF_W2 + row * HID + col : OFF_B2 + col;
}
}  // namespace net

// Device fields are pitched like the state: element (m, n) at
// (n - y1) * pitch + (m - x1 + xoff).
struct Args {
    const double *fld[5];          // u, v, ssh (current level), rest depth H, Coriolis rlh_s
    const double *fac[2];          // hu * dxt * dyh at ocean u points, hv * dyt * dxh at ocean v points, else 0
    const double *base[2];         // RHSx, RHSy without the closure
    double *out[2];                // RHSx, RHSy the substeps read
    void *feat;                    // features: BF16 [ny][nx][48], row n-ny0, column m-mx0
    const float *prm;              // FP32 parameter block (biases)
    const void *wb;                // BF16 weights
    long long pitch;
    int x1, x2, y1, y2, xoff;      // array bounds (bnd_*) and padding columns
    int mx0, mx1, ny0, ny1;        // interior
    float mean[5], inv_std[5];     // feature normalisation per field
    float out_scale[2];            // tendency (m/s^2) per unit network output
};

// out[c] = base[c] + y_c * out_scale[c] * fac[c] at the points where fac != 0
int apply(const Args &a, int nsm, cudaStream_t s);
// feat = the 48 features of every interior cell
int features(const Args &a, int nsm, cudaStream_t s);
// fac[0], fac[1] from the rest depth, the u/v masks and the metrics
int factors(const Args &a, const float *lcu, const float *lcv, const double *dxt, const double *dyh,
            const double *dyt, const double *dxh, double *fac_u, double *fac_v, cudaStream_t s);

// The training gradient on the tcgen05 tensor cores (closure_tc.cu):
// per-CTA partial sums (INMSOM_MLP_PARTIAL floats each) of grid persistent
// CTAs, grad_tc_ctas_per_sm per SM at most, over the batch's tiles of 128 samples;
// grad_tc_setup sets the kernel's shared-memory size once.
size_t grad_tc_smem();
int grad_tc_ctas_per_sm();
int grad_tc_setup();
int grad_tc(const void *x, const float *targets, const int *idx, int batch, const float *params, const void *wbf16,
            float *partial, int grid, cudaStream_t s);

}  // namespace closure
}  // namespace inmsom
