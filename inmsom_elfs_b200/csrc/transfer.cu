// Copies between the host's contiguous Fortran arrays and the pitched
// device arrays.
//
// The copy engine spends about 0.11-0.15 us on every row of a pitched copy,
// whatever its length: below 8 KB of row that, not the link, sets the time
// (3.1 KB rows moved at 28 GB/s, 0.8 KB rows at 7).  Such rows travel packed:
// the host side of a run of rows is contiguous per level, so one copy of few
// long pieces brings it to a packed stage on the device, and one kernel for
// all fields moves it into the pitched rows (or out of them), at HBM speed.
// Longer rows are copied pitched, which needs neither the stage nor the
// extra pass over memory (16 KB rows: 51 GB/s of the link's 55).
#include "transfer.h"

#include <algorithm>

namespace inmsom {
namespace transfer {

namespace {

constexpr size_t PACK_BELOW = 8192;          // bytes per row
constexpr size_t GROUP_BYTES = 64u << 20;    // a stage is reused after about this much
constexpr int MAX_FIELDS = 16;               // fields per kernel launch
constexpr int WARPS = 8;

struct Batch {
    void *dev[MAX_FIELDS];
    size_t off[MAX_FIELDS];    // in the stage
    int nlev[MAX_FIELDS], elem[MAX_FIELDS];
};

// one warp per row: field blockIdx.y, row w of nlev * nrows
template <bool UP>
__global__ void __launch_bounds__(32 * WARPS) k_rows(Dom d, const __grid_constant__ Batch b, unsigned char *stage, int r0, int nrows)
{
    const int f = blockIdx.y, lane = threadIdx.x & 31;
    const int nxa = d.bnd_x2 - d.bnd_x1 + 1, nya = d.bnd_y2 - d.bnd_y1 + 1;
    const long long total = (long long)b.nlev[f] * nrows;
    for (long long w = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5); w < total; w += (long long)gridDim.x * WARPS) {
        const long long lev = w / nrows;
        const long long at = (lev * nya + r0 + (w - lev * nrows)) * d.pitch + d.xoff;
        auto move = [&](auto *pitched, auto *packed) {
            for (int x = lane; x < nxa; x += 32) {
                if (UP) pitched[x] = packed[x];
                else packed[x] = pitched[x];
            }
        };
        if (b.elem[f] == 8)
            move(reinterpret_cast<double *>(b.dev[f]) + at, reinterpret_cast<double *>(stage + b.off[f]) + w * nxa);
        else
            move(reinterpret_cast<float *>(b.dev[f]) + at, reinterpret_cast<float *>(stage + b.off[f]) + w * nxa);
    }
}

cudaError_t reserve(Stage &st, size_t bytes)
{
    if (bytes <= st.cap) return cudaSuccess;
    release(st);
    const cudaError_t e = cudaMalloc(&st.p, bytes);
    if (e == cudaSuccess) st.cap = bytes;
    else st.p = nullptr;
    return e;
}

// one field's rows between the host and its place in the stage
cudaError_t packed_copy(unsigned char *stage, const Dom &d, const Field &f, int r0, int nrows, bool up, cudaStream_t s)
{
    const size_t row = (size_t)d.nxa() * f.elem, slab = row * nrows, level = row * d.nya();
    unsigned char *host = (unsigned char *)f.host + row * r0;
    const cudaMemcpyKind kind = up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    auto one = [&](size_t dev_off, size_t host_off, size_t bytes) {
        return up ? cudaMemcpyAsync(stage + dev_off, host + host_off, bytes, kind, s)
                  : cudaMemcpyAsync(host + host_off, stage + dev_off, bytes, kind, s);
    };
    if (slab == level || f.nlev == 1) return one(0, 0, slab * f.nlev);
    if (level < (size_t)1 << 31)   // the largest pitch of a 2-D copy
        return up ? cudaMemcpy2DAsync(stage, slab, host, level, slab, f.nlev, kind, s)
                  : cudaMemcpy2DAsync(host, level, stage, slab, slab, f.nlev, kind, s);
    for (int k = 0; k < f.nlev; k++) {
        const cudaError_t e = one(slab * k, level * k, slab);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t pitched_copy(const Dom &d, const Field &f, int r0, int nrows, bool up, cudaStream_t s)
{
    const size_t w = (size_t)d.nxa() * f.elem, pitch = (size_t)d.pitch * f.elem;
    const cudaMemcpyKind kind = up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    unsigned char *dev = (unsigned char *)f.dev + (size_t)d.xoff * f.elem, *host = (unsigned char *)f.host;
    if (nrows == d.nya() || f.nlev == 1) {   // consecutive levels' rows follow each other
        dev += pitch * r0;
        host += w * r0;
        const size_t h = (size_t)nrows * f.nlev;
        return up ? cudaMemcpy2DAsync(dev, pitch, host, w, w, h, kind, s)
                  : cudaMemcpy2DAsync(host, w, dev, pitch, w, h, kind, s);
    }
    cudaMemcpy3DParms p = {};
    const cudaPitchedPtr hp = make_cudaPitchedPtr(host, w, w, (size_t)d.nya());
    const cudaPitchedPtr dp = make_cudaPitchedPtr(dev, pitch, w, (size_t)d.nya());
    p.srcPtr = up ? hp : dp;
    p.dstPtr = up ? dp : hp;
    p.srcPos = p.dstPos = make_cudaPos(0, (size_t)r0, 0);
    p.extent = make_cudaExtent(w, (size_t)nrows, (size_t)f.nlev);
    p.kind = kind;
    return cudaMemcpy3DAsync(&p, s);
}

}  // namespace

cudaError_t rows(Stage &st, const Dom &d, const Field *f, int n, int r0, int r1, bool up, cudaStream_t s)
{
    const int nrows = r1 - r0 + 1;
    if (nrows < 1) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < n && e == cudaSuccess;) {
        if ((size_t)d.nxa() * f[k].elem >= PACK_BELOW) {
            e = pitched_copy(d, f[k++], r0, nrows, up, s);
            continue;
        }
        Batch b = {};
        size_t bytes = 0;
        int m = 0, tall = 1;
        for (; k + m < n && m < MAX_FIELDS && (m == 0 || bytes < GROUP_BYTES); m++) {
            const Field &g = f[k + m];
            if ((size_t)d.nxa() * g.elem >= PACK_BELOW) break;
            b.dev[m] = g.dev;
            b.off[m] = bytes;
            b.nlev[m] = g.nlev;
            b.elem[m] = g.elem;
            tall = std::max(tall, g.nlev);
            bytes += ((size_t)d.nxa() * g.elem * nrows * g.nlev + 255) / 256 * 256;
        }
        if ((e = reserve(st, bytes)) != cudaSuccess) break;
        unsigned char *stage = (unsigned char *)st.p;
        const dim3 grid((unsigned)std::min<long long>(((long long)nrows * tall + WARPS - 1) / WARPS, 1 << 16), m);
        if (!up) k_rows<false><<<grid, 32 * WARPS, 0, s>>>(d, b, stage, r0, nrows);
        for (int q = 0; q < m && e == cudaSuccess; q++) e = packed_copy(stage + b.off[q], d, f[k + q], r0, nrows, up, s);
        if (up && e == cudaSuccess) k_rows<true><<<grid, 32 * WARPS, 0, s>>>(d, b, stage, r0, nrows);
        if (e == cudaSuccess) e = cudaGetLastError();
        k += m;
    }
    return e;
}

void release(Stage &st)
{
    cudaFree(st.p);
    st = Stage{};
}

}  // namespace transfer
}  // namespace inmsom
