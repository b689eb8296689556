// Copies between the host's contiguous Fortran arrays and the pitched
// device arrays (see transfer.cu).
#pragma once

#include <cstddef>

#include "common.cuh"

namespace inmsom {
namespace transfer {

// one field: device base of its first level (pitched rows, levels pitch *
// rows apart), host array (bnd_x1:bnd_x2, bnd_y1:bnd_y2, nlev), bytes per
// element (4 or 8)
struct Field {
    void *dev;
    void *host;
    int nlev, elem;
};

// packed device copy of rows on their way up; owned by a context, used on one
// stream, grown to STAGE_BYTES at most: more than that goes through it in
// several turns (a turn costs a kernel launch, some microseconds against the
// millisecond that 64 MB take on the host link)
constexpr size_t STAGE_BYTES = 64u << 20;
constexpr int MAX_PIECES = 16;   // fields, or pieces of them, in a stage at once
struct Stage {
    void *p = nullptr;
    size_t cap = 0;
    size_t limit = STAGE_BYTES;
    int allocs = 0;              // allocations so far
};

// what an upload of nrows rows of n fields has in a stage at once
size_t packed_bytes(const Dom &d, const Field *f, int n, int nrows);
// room for `bytes`, as far as the limit and the device's memory go: a stage
// that cannot grow stays as it is.  Growing waits for the device, so that a
// caller who knows what is to come reserves it first
cudaError_t reserve(Stage &st, size_t bytes);

// rows r0..r1 (0-based from bnd_y1), whole rows of every level of n fields,
// to the device or to the host, enqueued on s
cudaError_t upload(Stage &st, const Dom &d, const Field *f, int n, int r0, int r1, cudaStream_t s);
cudaError_t download(const Dom &d, const Field *f, int n, int r0, int r1, cudaStream_t s);
void release(Stage &st);

}  // namespace transfer
}  // namespace inmsom
