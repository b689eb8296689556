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
// extra pass over memory (16 KB rows: 51 GB/s of the link's 55); so are all
// rows when the device has no memory left for a stage.
#include "transfer.h"

#include <algorithm>

namespace inmsom {
namespace transfer {

namespace {

constexpr size_t PACK_BELOW = 8192;          // bytes per row
constexpr int MAX_PIECES = 16;               // pieces per kernel launch
constexpr int WARPS = 8;

// pieces of fields: nrows rows from r0 on of nlev levels each
struct Batch {
    void *dev[MAX_PIECES];     // row 0 of the piece's first level
    size_t off[MAX_PIECES];    // in the stage
    int nlev[MAX_PIECES], elem[MAX_PIECES], r0[MAX_PIECES], nrows[MAX_PIECES];
};

// one warp per row: piece blockIdx.y, row w of nlev * nrows
template <bool UP>
__global__ void __launch_bounds__(32 * WARPS) k_rows(Dom d, const __grid_constant__ Batch b, unsigned char *stage)
{
    const int f = blockIdx.y, lane = threadIdx.x & 31, r0 = b.r0[f], nrows = b.nrows[f];
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

size_t padded(size_t bytes) { return (bytes + 255) / 256 * 256; }

// a piece's rows between the host and its place in the stage
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

size_t packed_bytes(const Dom &d, const Field *f, int n, int nrows)
{
    size_t bytes = 0;
    for (int k = 0; k < n; k++) {
        const size_t line = (size_t)d.nxa() * f[k].elem;
        if (line < PACK_BELOW) bytes += padded(line * nrows * f[k].nlev);
    }
    return bytes;
}

cudaError_t reserve(Stage &st, size_t bytes)
{
    bytes = std::min(bytes, st.limit);
    if (bytes <= st.cap) return cudaSuccess;
    void *p = nullptr;
    const cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        return cudaSuccess;
    }
    if (e != cudaSuccess) return e;
    release(st);
    st.p = p;
    st.cap = bytes;
    st.allocs++;
    return cudaSuccess;
}

cudaError_t rows(Stage &st, const Dom &d, const Field *f, int n, int r0, int r1, bool up, cudaStream_t s)
{
    const int nrows = r1 - r0 + 1;
    if (nrows < 1) return cudaSuccess;
    cudaError_t e = reserve(st, packed_bytes(d, f, n, nrows));
    int k = 0, lev = 0, row = r0;   // the next field, and the level and row it goes on with
    while (k < n && e == cudaSuccess) {
        const size_t line = (size_t)d.nxa() * f[k].elem;
        if (line >= PACK_BELOW || line > st.cap) {
            e = pitched_copy(d, f[k++], r0, nrows, up, s);
            continue;
        }
        // fill the stage: whole fields, and of one too large for it runs of
        // levels (or of a level's rows)
        Batch b = {};
        Field part[MAX_PIECES];
        size_t used = 0;
        int m = 0;
        long long tall = 1;
        for (; k < n && m < MAX_PIECES; m++) {
            const Field &g = f[k];
            const size_t line = (size_t)d.nxa() * g.elem, slab = line * nrows, room = st.cap - used;
            if (line >= PACK_BELOW || line > st.cap) break;
            int levels = g.nlev - lev, lines = nrows;
            if (row != r0 || slab * levels > room) {
                if (m > 0) break;
                if (row == r0 && slab <= room) {
                    levels = (int)(room / slab);
                } else {
                    levels = 1;
                    lines = (int)std::min<size_t>(r1 - row + 1, room / line);
                }
            }
            const size_t above = (size_t)lev * d.nya();   // rows of the levels before
            part[m] = Field{(unsigned char *)g.dev + above * d.pitch * g.elem, (unsigned char *)g.host + above * line, levels,
                            g.elem};
            b.dev[m] = part[m].dev;
            b.off[m] = used;
            b.nlev[m] = levels;
            b.elem[m] = g.elem;
            b.r0[m] = row;
            b.nrows[m] = lines;
            tall = std::max(tall, (long long)levels * lines);
            used = std::min(st.cap, used + padded(line * lines * levels));
            if (lines == nrows) {
                lev += levels;
            } else if ((row += lines) > r1) {
                row = r0;
                lev++;
            }
            if (lev == g.nlev) {
                lev = 0;
                k++;
            }
        }
        unsigned char *stage = (unsigned char *)st.p;
        const dim3 grid((unsigned)std::min<long long>((tall + WARPS - 1) / WARPS, 1 << 16), m);
        if (!up) k_rows<false><<<grid, 32 * WARPS, 0, s>>>(d, b, stage);
        for (int q = 0; q < m && e == cudaSuccess; q++) e = packed_copy(stage + b.off[q], d, part[q], b.r0[q], b.nrows[q], up, s);
        if (up && e == cudaSuccess) k_rows<true><<<grid, 32 * WARPS, 0, s>>>(d, b, stage);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    return e;
}

void release(Stage &st)
{
    cudaFree(st.p);
    st.p = nullptr;
    st.cap = 0;
}

}  // namespace transfer
}  // namespace inmsom
