// Copies between the host's contiguous Fortran arrays and the pitched
// device arrays.
//
// Downloads are pitched copies, which run at the link's rate for rows of any
// length (42-50 GB/s of 55), and so are uploads of rows that are a multiple of
// 128 bytes.  On other rows of an upload the copy engine spends 0.11-0.15 us
// each, whatever their length: below 8 KB of row that, not the link, sets the
// time (3.1 KB rows moved at 28 GB/s, 0.8 KB rows at 7).  Such rows travel
// packed: the host side of a run of rows is contiguous per level, so one copy
// of few long pieces brings it to a packed stage on the device, and one kernel
// for all fields moves it into the pitched rows, at HBM speed.  A field that
// is uploaded alone waits for that kernel and gains less: it is packed below
// 4 KB of row.  us per call, all rows pitched and so packed: the barotropic
// call with every array in and out (21 fields up, 19 down) on 200 x 150 points
// (1632-byte rows) 729, 526, on 1015 x 400 (8152 bytes) 3004, 2803, on
// 300 x 200 (2432 bytes, 19 x 128) 671, 669, but 690 with those packed too and
// 716 with the downloads packed as well; baroclinic_dynamics on 512 x 384 x 20
// 11962, 8502, on 508 x 384 x 20 (4096-byte rows) 7518, 7470, packed 7906; one
// field up and down on 400 x 300 79, 73, on 800 x 300 (6432 bytes) 113, 113,
// packed 120.  All rows are copied pitched when the device has no memory left
// for a stage.
#include "transfer.h"

#include <algorithm>

namespace inmsom {
namespace transfer {

namespace {

constexpr int WARPS = 8;

// bytes per row of a field, and whether it is packed as one of n
size_t line_of(const Dom &d, const Field &f) { return (size_t)d.nxa() * f.elem; }
bool packs(const Dom &d, const Field &f, int n)
{
    const size_t line = line_of(d, f);
    return line % 128 != 0 && line < (n == 1 && f.nlev == 1 ? 4096u : 8192u);
}

// pieces of fields: nrows rows from r0 on of nlev levels each
struct Batch {
    void *dev[MAX_PIECES];     // row 0 of the piece's first level
    size_t off[MAX_PIECES];    // in the stage
    int nlev[MAX_PIECES], elem[MAX_PIECES], r0[MAX_PIECES], nrows[MAX_PIECES];
};

// one warp per row: piece blockIdx.y, row w of nlev * nrows
__global__ void __launch_bounds__(32 * WARPS) k_unpack(Dom d, const __grid_constant__ Batch b, const unsigned char *stage)
{
    const int f = blockIdx.y, lane = threadIdx.x & 31, r0 = b.r0[f], nrows = b.nrows[f];
    const int nxa = d.bnd_x2 - d.bnd_x1 + 1, nya = d.bnd_y2 - d.bnd_y1 + 1;
    const long long total = (long long)b.nlev[f] * nrows;
    for (long long w = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5); w < total; w += (long long)gridDim.x * WARPS) {
        const long long lev = w / nrows;
        const long long at = (lev * nya + r0 + (w - lev * nrows)) * d.pitch + d.xoff;
        auto move = [&](auto *pitched, auto *packed) {
            for (int x = lane; x < nxa; x += 32) pitched[x] = packed[x];
        };
        if (b.elem[f] == 8)
            move(reinterpret_cast<double *>(b.dev[f]) + at, reinterpret_cast<const double *>(stage + b.off[f]) + w * nxa);
        else
            move(reinterpret_cast<float *>(b.dev[f]) + at, reinterpret_cast<const float *>(stage + b.off[f]) + w * nxa);
    }
}

size_t padded(size_t bytes) { return (bytes + 255) / 256 * 256; }

// a piece's rows from the host to its place in the stage
cudaError_t packed_copy(unsigned char *stage, const Dom &d, const Field &f, int r0, int nrows, cudaStream_t s)
{
    const size_t row = line_of(d, f), slab = row * nrows, level = row * d.nya();
    const unsigned char *host = (const unsigned char *)f.host + row * r0;
    if (slab == level || f.nlev == 1) return cudaMemcpyAsync(stage, host, slab * f.nlev, cudaMemcpyHostToDevice, s);
    if (level < (size_t)1 << 31)   // the largest pitch of a 2-D copy
        return cudaMemcpy2DAsync(stage, slab, host, level, slab, f.nlev, cudaMemcpyHostToDevice, s);
    for (int k = 0; k < f.nlev; k++) {
        const cudaError_t e = cudaMemcpyAsync(stage + slab * k, host + level * k, slab, cudaMemcpyHostToDevice, s);
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
    size_t most = 0, bytes[MAX_PIECES] = {};
    for (int k = 0, at = 0; k < n; k++) {   // the last MAX_PIECES packed fields
        if (!packs(d, f[k], n)) continue;
        bytes[at] = padded(line_of(d, f[k]) * nrows * f[k].nlev);
        at = (at + 1) % MAX_PIECES;
        size_t sum = 0;
        for (size_t b : bytes) sum += b;
        most = std::max(most, sum);
    }
    return most;
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

cudaError_t upload(Stage &st, const Dom &d, const Field *f, int n, int r0, int r1, cudaStream_t s)
{
    const int nrows = r1 - r0 + 1;
    if (nrows < 1) return cudaSuccess;
    cudaError_t e = reserve(st, packed_bytes(d, f, n, nrows));
    int k = 0, lev = 0, row = r0;   // the next field, and the level and row it goes on with
    while (k < n && e == cudaSuccess) {
        if (!packs(d, f[k], n) || line_of(d, f[k]) > st.cap) {
            e = pitched_copy(d, f[k++], r0, nrows, true, s);
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
            const size_t line = line_of(d, g), slab = line * nrows, room = st.cap - used;
            if (!packs(d, g, n) || line > st.cap) break;
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
        for (int q = 0; q < m && e == cudaSuccess; q++) e = packed_copy(stage + b.off[q], d, part[q], b.r0[q], b.nrows[q], s);
        if (e != cudaSuccess) break;
        k_unpack<<<grid, 32 * WARPS, 0, s>>>(d, b, stage);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t download(const Dom &d, const Field *f, int n, int r0, int r1, cudaStream_t s)
{
    if (r1 < r0) return cudaSuccess;
    for (int k = 0; k < n; k++) {
        const cudaError_t e = pitched_copy(d, f[k], r0, r1 - r0 + 1, false, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void release(Stage &st)
{
    cudaFree(st.p);
    st.p = nullptr;
    st.cap = 0;
}

}  // namespace transfer
}  // namespace inmsom
