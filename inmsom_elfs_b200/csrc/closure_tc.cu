// Training gradient of the closure MLP (45 -> 64 -> 64 -> 2, GELU, mean
// squared error) on the fifth-generation tensor cores: tcgen05.mma with
// BF16 operands in shared memory and FP32 accumulators in tensor memory.
// No counterpart in the reference (the closure stands in for the Laplacian
// viscosity of uv_diff2, Function/vel_ssh.f90:117-184, on coarse grids).
//
// Two CTAs of eight warps per SM, each persistent over tiles of 128 samples.
// A tile is a chain of small MMA groups and elementwise phases, bound by the
// latency of its steps (the tensor pipe is a few per cent busy), so that a
// second CTA on the SM runs in the first one's waits.  Warp w reads
// tensor-memory lanes 32 (w % 4) .. +31 (the lane quarter it may access), so
// each thread owns one sample (its lane) and 32 of the 64 columns of every
// layer's output (w / 4 picks which); the next tile's inputs are fetched
// while a tile computes.  One thread issues the MMAs.  Per tile:
//   forward   Z1 = X W1, A1 = GELU(Z1 + b1); Z2 = A1 W2, A2 = GELU(Z2 + b2);
//             O = A2 W3 (+ b3)                        (M = 128 samples)
//   backward  D3 = 2 (O - T) / (batch * 2); DA2 = D3 W3^T;
//             DZ2 = DA2 * GELU'(Z2 + b2); DA1 = DZ2 W2^T;
//             DZ1 = DA1 * GELU'(Z1 + b1)               (M = 128 samples)
//   weights   dW3 += A2^T D3, dW2 += A1^T DZ2, dW1 += X^T DZ1
//             (M = the layer's inputs, K = the tile's samples), accumulated
//             in tensor memory over all tiles of the CTA.
// GELU' of both layers stays in the thread's registers from the forward
// phase, so that one block of 64 tensor-memory columns serves Z1, Z2, O, DA2
// and DA1 in turn (208 columns with the weight gradients: two CTAs' worth
// fit), and DZ2, DZ1 go over A2, A1 in shared memory once those are used up
// (86 KB).  A tile's dW1 is issued with the next tile's Z1 (X has two
// buffers): five steps per tile, one barrier and one wait each.  Measured
// (gradient, reduction and Adam): 24.4 us per training step at batch 65536,
// 12.0 at 1024, against 42.0 and 22.6 with one CTA of sixteen warps, seven
// steps per tile and the partial sums stored row by row.  The two CTAs leave
// 128 registers per thread, of which the compiler spills 18 bytes.
// The bias gradients come out of the same weight-gradient products: X, A1
// and A2 carry a column of ones (X column 48, A1/A2 column 64), whose row
// of dW is the column sum of the layer's output gradient.
//
// Shared-memory operands use the no-swizzle canonical layout of the
// tensor-core descriptors: 8 x 16-byte core matrices, element (r, c) of an
// R x C tile at ((r / 8) * (C / 8) + c / 8) * 128 + (r % 8) * 16 +
// (c % 8) * 2 bytes.  Read with rows as M/N and columns as K (K-major) it
// is the forward operand; read with columns as M/N and rows as K (MN-major)
// the same bytes are its transpose, so no tile is ever transposed.
//
// Every mbarrier wait is bounded; a wait that gives up makes the CTA's
// partial sums NaN (the gradient and the loss come out NaN), and the CTA
// frees its tensor memory and returns.
#include "inmsom_gpu.h"
#include "closure.h"
#include "gelu.cuh"

#include <cuda_bf16.h>

#include <cstddef>
#include <cstdint>

namespace {

using namespace inmsom::closure;

using namespace inmsom::closure::net;
constexpr int BOFF_W1 = 0, BOFF_W2 = KIN * HID, BOFF_W3 = BOFF_W2 + HID * HID;
static_assert(NPARAM == INMSOM_MLP_NPARAM, "parameter block size");
constexpr int NPART = NPARAM + 1;
constexpr int TILE = 128, THREADS = 256, CTAS_PER_SM = 2;
constexpr int SLICE = 32;                 // columns of a 64-column block per thread (2 warps per lane quarter)
constexpr int NO = 16;                    // output columns of the MMAs (2 used)
// columns of the X and A1/A2 tiles: the data, then a group of eight with the
// ones column.  The weight-gradient products read 64 (X) and 128 (A1, A2)
// columns as their M: what they read past the tile's columns (the next rows
// of the tile, or the buffer after it) only reaches rows of dW that are
// never read
constexpr int XC = 56, AC = 72;
constexpr unsigned WAIT_POLLS = 1u << 24;

// tensor-memory columns (256 allocated: two CTAs per SM)
constexpr uint32_t TM_COLS = 256;
constexpr uint32_t C_W = 0, C_DW1 = 64, C_DW2 = 128, C_DW3 = 192;
static_assert(C_DW3 + NO <= TM_COLS, "tensor-memory columns");

struct __align__(128) Smem {
    __nv_bfloat16 x[2][TILE * XC];   // inputs, column 48 = 1
    __nv_bfloat16 a1[TILE * AC];     // GELU(Z1 + b1), column 64 = 1; then DZ1 in columns 0..63
    __nv_bfloat16 a2[TILE * AC];     // GELU(Z2 + b2), column 64 = 1; then DZ2 in columns 0..63
    __nv_bfloat16 w1[KIN * HID];     // rows = inputs, columns = outputs, as in the parameter block
    __nv_bfloat16 w2[HID * HID];
    __nv_bfloat16 w3[HID * NO];      // 16 outputs (2 used)
    __nv_bfloat16 d3[TILE * NO];
    float b1[HID], b2[HID], b3[NO];
    float loss[4];
    uint64_t mbar;
    uint32_t tmem_base;
};
// bytes a descriptor may reach past a2 (its last rows, columns 72..127) stay
// inside the structure
static_assert(sizeof(Smem) - offsetof(Smem, w1) >= (128 - AC) * 16, "operand reads stay in the structure");

// element (r, c) of an R x C tile with C columns, in elements
__device__ __forceinline__ int blk(int r, int c, int C) { return ((r >> 3) * (C >> 3) + (c >> 3)) * 64 + (r & 7) * 8 + (c & 7); }

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, no swizzle: lbo / sbo in bytes
__device__ __forceinline__ uint64_t sdesc(const void *p, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr(p) >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor of kind::f16: BF16 A and B, FP32 D
__host__ __device__ constexpr uint32_t idesc(int M, int N, bool a_mn, bool b_mn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ void commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
                 : "memory");
}

__device__ __forceinline__ bool wait_bar(uint64_t *bar, uint32_t parity)
{
    for (unsigned i = 0; i < WAIT_POLLS; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(saddr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_smem_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 or 32 consecutive FP32 columns of this thread's tensor-memory lane.  The
// load fills its registers some time after it is issued: its wait is part of
// the same statement, so that no use of them can be placed between the two
__device__ __forceinline__ void ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = __uint_as_float(r[k]);
}
__device__ __forceinline__ void ld32(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int k = 0; k < 32; k++) v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// 8 consecutive values as one 16-byte chunk of row r of a tile
__device__ __forceinline__ void st_chunk(__nv_bfloat16 *tile, int r, int c0, int C, const float *v)
{
    const uint4 q = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
    *reinterpret_cast<uint4 *>(tile + blk(r, c0, C)) = q;
}

__global__ void __launch_bounds__(THREADS, CTAS_PER_SM)
    k_mlp_grad_tc(const __nv_bfloat16 *__restrict__ x, const float *__restrict__ tgt, const int *__restrict__ idx,
                  int batch, const float *__restrict__ prm, const __nv_bfloat16 *__restrict__ wb,
                  float *__restrict__ partial)
{
    extern __shared__ __align__(1024) unsigned char raw[];
    Smem &s = *reinterpret_cast<Smem *>(raw);
    const int t = threadIdx.x, w = t >> 5, q = w & 3, cs = w >> 2;
    const int r = 32 * q + (t & 31);       // this thread's sample row and tensor-memory lane
    const int c0 = SLICE * cs;             // its columns of a 64-column block
    const bool issuer = t == 0;
    const int ntiles = batch / TILE;

    // this thread's part of a sample: 16-byte chunks 3 cs .. 3 cs + 2 (of 6),
    // and (slice 0) the two targets
    uint4 xa[3];
    float t0 = 0.f, t1 = 0.f;
    auto fetch = [&](int tile) {
        if (tile >= ntiles) return;
        const long long row = idx ? (long long)idx[tile * TILE + r] : (long long)tile * TILE + r;
        const uint4 *src = reinterpret_cast<const uint4 *>(x + row * KIN) + 3 * cs;
#pragma unroll
        for (int k = 0; k < 3; k++) xa[k] = src[k];
        if (cs == 0) {
            t0 = tgt[row * NOUT];
            t1 = tgt[row * NOUT + 1];
        }
    };
    if (issuer) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&s.mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // Launched with programmatic stream serialisation: what follows reads what
    // earlier kernels of the stream wrote (the weights, the batch).  The
    // tensor memory is taken after it too, while the first loads are under
    // way: the stream's last kernel may be another program's that takes
    // tensor memory after it let this one in, and would wait for columns held
    // by a CTA that waits for its end.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    fetch(blockIdx.x);
    // weights, 16 bytes (8 outputs of one input) at a time
    {
        constexpr int G = HID / 8, N1 = KIN * G, N2 = HID * G;   // pieces
        static_assert(N1 <= 2 * THREADS && N2 <= 2 * THREADS && HID <= THREADS, "pieces per thread");
        const uint4 *w16 = reinterpret_cast<const uint4 *>(wb);
        uint4 p1[2] = {}, p2[2] = {}, p3 = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = t + h * THREADS;
            if (i < N1) p1[h] = w16[(BOFF_W1 / 8) + i];
            if (i < N2) p2[h] = w16[(BOFF_W2 / 8) + i];
        }
        if (t < HID) p3 = w16[(BOFF_W3 / 8) + t];
        if (w == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&s.tmem_base)),
                         "r"(TM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = t + h * THREADS;
            if (i < N1) *reinterpret_cast<uint4 *>(s.w1 + blk(i / G, 8 * (i % G), HID)) = p1[h];
            if (i < N2) *reinterpret_cast<uint4 *>(s.w2 + blk(i / G, 8 * (i % G), HID)) = p2[h];
        }
        if (t < HID) {
            *reinterpret_cast<uint4 *>(s.w3 + blk(t, 0, NO)) = p3;
            *reinterpret_cast<uint4 *>(s.w3 + blk(t, 8, NO)) = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    if (t < HID) {
        s.b1[t] = prm[OFF_B1 + t];
        s.b2[t] = prm[OFF_B2 + t];
    }
    if (t < NO) s.b3[t] = t < N3 ? prm[OFF_B3 + t] : 0.f;
    {
        float one[8] = {1.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        st_chunk(s.x[cs], r, KIN, XC, one);
        if (cs == 0) {
            st_chunk(s.a1, r, HID, AC, one);
            st_chunk(s.d3, r, 8, NO, zero);
        } else {
            st_chunk(s.a2, r, HID, AC, one);
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tb = s.tmem_base;
    const uint32_t lane = tb + ((uint32_t)(32 * q) << 16);   // this warp's lane quarter
    const float scale = 2.0f / ((float)batch * NOUT);
    uint32_t ph = 0;
    float lsum = 0.f;
    bool got = true, ok = true, first = true;

    // all threads: shared-memory writes visible to the tensor cores and
    // tensor-memory reads done before the issuer's next MMAs; false (for
    // every thread) if some thread's last wait gave up
    auto handoff = [&]() -> bool {
        fence_smem_async();
        fence_before();
        ok = __syncthreads_or(!got) == 0;
        fence_after();
        return ok;
    };
    // the issuer's MMAs so far, waited for by every thread
    auto finish = [&]() {
        if (issuer) commit(&s.mbar);
        got = wait_bar(&s.mbar, ph);
        ph ^= 1u;
        fence_after();
    };
    auto put_x = [&](int buf) {
#pragma unroll
        for (int k = 0; k < 3; k++) *reinterpret_cast<uint4 *>(s.x[buf] + blk(r, 8 * (3 * cs + k), XC)) = xa[k];
    };
    // dW1 += X^T DZ1 (M = 64 columns of X) of the tile in buffer buf
    auto issue_dw1 = [&](int buf, bool fresh) {
        for (int ks = 0; ks < 8; ks++)
            mma(tb + C_DW1, sdesc(s.x[buf] + ks * 16 * XC, XC * 16, 128), sdesc(s.a1 + ks * 16 * AC, AC * 16, 128),
                idesc(64, 64, true, true), !(fresh && ks == 0));
    };
    // a layer's activations from its accumulator: GELU to the operand tile,
    // GELU' kept
    auto activate = [&](const float *bias, __nv_bfloat16 *tile, float (&d)[SLICE]) {
        float z[SLICE];
        ld32(lane + C_W + c0, z);
#pragma unroll
        for (int k = 0; k < SLICE; k++) gelu_both(z[k] + bias[c0 + k], z[k], d[k]);
#pragma unroll
        for (int k = 0; k < SLICE; k += 8) st_chunk(tile, r, c0 + k, AC, z + k);
    };
    // a layer's pre-activation gradient from the accumulator
    auto backward = [&](__nv_bfloat16 *tile, const float (&d)[SLICE]) {
        float da[SLICE];
        ld32(lane + C_W + c0, da);
#pragma unroll
        for (int k = 0; k < SLICE; k++) da[k] *= d[k];
#pragma unroll
        for (int k = 0; k < SLICE; k += 8) st_chunk(tile, r, c0 + k, AC, da + k);
    };

    int buf = 0;
    if (blockIdx.x < ntiles) put_x(0);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, buf ^= 1) {
        // X (and the last tile's DZ1) are in place
        const float tg0 = t0, tg1 = t1;
        if (!handoff()) break;
        // ---- the last tile's dW1; Z1 = X W1 (K = 48)
        if (issuer) {
            if (!first) issue_dw1(buf ^ 1, tile == blockIdx.x + gridDim.x);
            for (int ks = 0; ks < 3; ks++)
                mma(tb + C_W, sdesc(s.x[buf] + 128 * ks, 128, XC * 16), sdesc(s.w1 + ks * 16 * HID, 1024, 128),
                    idesc(128, 64, false, true), ks > 0);
        }
        fetch(tile + gridDim.x);
        finish();
        float d1[SLICE], d2[SLICE];
        activate(s.b1, s.a1, d1);
        if (!handoff()) break;
        // ---- Z2 = A1 W2 (K = 64)
        if (issuer)
            for (int ks = 0; ks < 4; ks++)
                mma(tb + C_W, sdesc(s.a1 + 128 * ks, 128, AC * 16), sdesc(s.w2 + ks * 16 * HID, 1024, 128),
                    idesc(128, 64, false, true), ks > 0);
        finish();
        activate(s.b2, s.a2, d2);
        if (!handoff()) break;
        // ---- O = A2 W3 (N = 16, 2 used)
        if (issuer)
            for (int ks = 0; ks < 4; ks++)
                mma(tb + C_W, sdesc(s.a2 + 128 * ks, 128, AC * 16), sdesc(s.w3 + ks * 16 * NO, 256, 128),
                    idesc(128, NO, false, true), ks > 0);
        finish();
        if (cs == 0) {
            float o[16];
            ld16(lane + C_W, o);
            const float e0 = o[0] + s.b3[0] - tg0, e1 = o[1] + s.b3[1] - tg1;
            lsum += e0 * e0 + e1 * e1;
            float d[8] = {scale * e0, scale * e1, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            st_chunk(s.d3, r, 0, NO, d);
        }
        if (!handoff()) break;
        // ---- DA2 = D3 W3^T (K = 16); dW3 += A2^T D3 (M = 128 columns of A2, K = 128 samples)
        if (issuer) {
            mma(tb + C_W, sdesc(s.d3, 128, 256), sdesc(s.w3, 128, 256), idesc(128, 64, false, false), 0);
            for (int ks = 0; ks < 8; ks++)
                mma(tb + C_DW3, sdesc(s.a2 + ks * 16 * AC, AC * 16, 128), sdesc(s.d3 + ks * 16 * NO, 256, 128),
                    idesc(128, NO, true, true), !(first && ks == 0));
        }
        finish();
        backward(s.a2, d2);
        if (!handoff()) break;
        // ---- DA1 = DZ2 W2^T (K = 64); dW2 += A1^T DZ2
        if (issuer) {
            for (int ks = 0; ks < 4; ks++)
                mma(tb + C_W, sdesc(s.a2 + 128 * ks, 128, AC * 16), sdesc(s.w2 + 128 * ks, 128, 1024),
                    idesc(128, 64, false, false), ks > 0);
            for (int ks = 0; ks < 8; ks++)
                mma(tb + C_DW2, sdesc(s.a1 + ks * 16 * AC, AC * 16, 128), sdesc(s.a2 + ks * 16 * AC, AC * 16, 128),
                    idesc(128, 64, true, true), !(first && ks == 0));
        }
        finish();
        backward(s.a1, d1);
        if (tile + gridDim.x < ntiles) put_x(buf ^ 1);
        first = false;
    }
    if (ok && !first && handoff()) {
        // ---- the last tile's dW1
        if (issuer) issue_dw1(buf ^ 1, blockIdx.x + gridDim.x >= ntiles);
        finish();
        ok = __syncthreads_or(!got) == 0;
        fence_after();
    }

    if (ok && !first) {
        // column by column (partial_param): the lanes of a warp hold
        // consecutive rows, so that a store is one run of addresses (row by
        // row, 32 separate sectors a store, took 10 of the kernel's 33 us)
        float *out = partial + (size_t)blockIdx.x * NPART;
        float v[SLICE];
        {
            // dW1: M = 64 rows in lanes 32 q + (0..15) of quarter q: row 16 q + lane
            const int lr = t & 31, m64 = 16 * q + lr;
            ld32(lane + C_DW1 + c0, v);
            if (lr < 16 && m64 < ROWS1)
#pragma unroll
                for (int k = 0; k < SLICE; k++) out[(c0 + k) * ROWS1 + m64] = v[k];
        }
        ld32(lane + C_DW2 + c0, v);
        if (r < ROWS2)
#pragma unroll
            for (int k = 0; k < SLICE; k++) out[PART_W2 + (c0 + k) * ROWS2 + r] = v[k];
        if (cs == 0) {
            float o[16];
            ld16(lane + C_DW3, o);
            if (r < ROWS2)
#pragma unroll
                for (int k = 0; k < N3; k++) out[PART_W3 + k * ROWS2 + r] = o[k];
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, m);
            if ((t & 31) == 0) s.loss[q] = lsum;
        }
        __syncthreads();
        if (t == 0) out[NPARAM] = (s.loss[0] + s.loss[1]) + (s.loss[2] + s.loss[3]);
    }
    if (!ok) {
        // a wait gave up: the CTA's partial sums are NaN (so the gradient
        // and the loss are), and the MMAs of the step that timed out are
        // waited for (bounded) before the tensor memory is freed
        float *out = partial + (size_t)blockIdx.x * NPART;
        for (int i = t; i < NPART; i += THREADS) out[i] = __int_as_float(0x7fc00000);
        if (issuer) (void)wait_bar(&s.mbar, ph ^ 1u);
    }
    fence_before();
    __syncthreads();
    if (w == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(TM_COLS) : "memory");
    }
}

}  // namespace

namespace inmsom {
namespace closure {

size_t grad_tc_smem() { return sizeof(Smem); }

int grad_tc_ctas_per_sm() { return CTAS_PER_SM; }

int grad_tc(const void *x, const float *targets, const int *idx, int batch, const float *params, const void *wbf16,
            float *partial, int grid, cudaStream_t s)
{
    return launch_after(k_mlp_grad_tc, grid, THREADS, grad_tc_smem(), s, (const __nv_bfloat16 *)x, targets, idx, batch,
                        params, (const __nv_bfloat16 *)wbf16, partial) != cudaSuccess;
}

int grad_tc_setup()
{
    return cudaFuncSetAttribute(k_mlp_grad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grad_tc_smem()) !=
           cudaSuccess;
}

}  // namespace closure
}  // namespace inmsom
