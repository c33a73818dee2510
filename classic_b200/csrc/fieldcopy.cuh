// Host arrays to and from the pitched device fields.
//
// A caller's array is dense [nfields][rows][width] doubles, usually pageable;
// the device rows are padded and may be FP32.  The driver copies a pageable 2D
// block row by row and field by field.  us for Euler's four fields, in / out of
// the device, against one dense copy to or from a device buffer with a kernel
// that lays the rows out: 72^2 57 / 62 against 30 / 34, 200^2 113 / 140 against
// 89 / 107, 384^2 327 / 367 against 270 / 275, 700^2 813 / 861 against 820 /
// 800.  So FP64 blocks of several fields take the buffer up to STAGE_BYTES.  A
// single field, a 1D grid and up to 64 KB in are cheaper directly (annulus
// 40x120: 28 against 38; 40^2 42 against 43 to 58; one unpadded field of 64^2
// 17 against 29 for a 1D copy), and where no row is padded the whole block is
// one copy (four of 128^2 out: 90 against 54).  FP32 blocks need the buffer for
// the conversion at any size; a single field of 24 to 64 KB goes into it as a 2D
// block too (64x128 22 against 51, 90x91 34 against 50; the other way 30x90, 21
// KB, 32 against 26, three fields of 45^2 61 against 41).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "host.h"

namespace clawb200 {

constexpr size_t STAGE_BYTES = 8u << 20;
constexpr size_t SMALL_IN = 64u << 10;

// The buffer of an object, n doubles.  Copies through it are two operations on
// the object's stream; `order` keeps them together, so that the stream's order
// keeps the copies of several host threads apart.
struct Stage {
    double* buf = nullptr;
    size_t n = 0;
    std::mutex order;
    ~Stage() {
        if (buf) cudaFree(buf);
    }
};

// A caller's dense block and its place on the device.
struct Block {
    long long pitch, fpitch;  // elements from row to row, from field to field
    int nfields;
    long long width, rows;
    size_t count() const { return (size_t)nfields * rows * width; }
    // whether the copy in (or out) takes the buffer; the FP64 rule is above
    bool staged(size_t elem, bool in) const {
        if (elem == 4) return true;
        const size_t bytes = count() * 8;
        const bool padded = pitch != width || fpitch != width * rows;
        return padded && nfields > 1 && rows > 1 && bytes <= STAGE_BYTES && !(in && bytes <= SMALL_IN);
    }
};

// one element a thread, rows over blockIdx.y; row r of field m is dense row
// m*rows + r
template <class real, bool IN>
__global__ void __launch_bounds__(256)
copy_rows(double* dense, real* dev, long long pitch, long long fpitch, long long width, long long rows,
          long long nrows) {
    const long long x = blockIdx.x * 256ll + threadIdx.x;
    if (x >= width) return;
    for (long long k = blockIdx.y; k < nrows; k += gridDim.y) {
        const long long m = k / rows, r = k - m * rows;
        real* d = dev + m * fpitch + r * pitch + x;
        if constexpr (IN) *d = (real)dense[k * width + x];
        else dense[k * width + x] = (double)*d;
    }
}

// Queue the copy of a block on the object's stream (the caller waits for it).
template <class real>
int copy_fields(real* dev, const Block& b, double* host, Stage& stage, bool in, cudaStream_t st) {
    const size_t n = b.count();
    const auto kind = in ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    if constexpr (sizeof(real) == 8) {
        const bool small_in = in && n * 8 <= SMALL_IN;
        if (b.pitch == b.width && b.fpitch == b.width * b.rows && !small_in) {
            if (in) CUDA_TRY(cudaMemcpyAsync(dev, host, n * 8, kind, st));
            else CUDA_TRY(cudaMemcpyAsync(host, dev, n * 8, kind, st));
            return 0;
        }
        if (!b.staged(8, in) || n > stage.n) {  // (no buffer where memory was short)
            for (int m = 0; m < b.nfields; ++m) {
                real* d = dev + m * b.fpitch;
                double* hp = host + (size_t)m * b.width * b.rows;
                if (in) CUDA_TRY(cudaMemcpy2DAsync(d, b.pitch * 8, hp, b.width * 8, b.width * 8, b.rows, kind, st));
                else CUDA_TRY(cudaMemcpy2DAsync(hp, b.width * 8, d, b.pitch * 8, b.width * 8, b.rows, kind, st));
            }
            return 0;
        }
    }
    const long long nrows = b.nfields * b.rows;
    const dim3 grid((unsigned)((b.width + 255) / 256), (unsigned)std::min(nrows, 65535ll));
    std::lock_guard<std::mutex> together(stage.order);
    if (in) {
        if (b.nfields == 1 && n * 8 > (24u << 10) && n * 8 <= SMALL_IN)
            CUDA_TRY(cudaMemcpy2DAsync(stage.buf, b.width * 8, host, b.width * 8, b.width * 8, b.rows, kind, st));
        else
            CUDA_TRY(cudaMemcpyAsync(stage.buf, host, n * 8, kind, st));
        copy_rows<real, true><<<grid, 256, 0, st>>>(stage.buf, dev, b.pitch, b.fpitch, b.width, b.rows, nrows);
    } else {
        copy_rows<real, false><<<grid, 256, 0, st>>>(stage.buf, dev, b.pitch, b.fpitch, b.width, b.rows, nrows);
        CUDA_TRY(cudaMemcpyAsync(host, stage.buf, n * 8, kind, st));
    }
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// The buffer for copies of up to n doubles (0: none takes it).  FP32 fields
// cannot do without (`needed`), FP64 ones can when memory is short.
inline int make_stage(Stage& stage, size_t n, bool needed) {
    if (!n) return 0;
    const cudaError_t e = cudaMalloc(&stage.buf, n * 8);
    if (e != cudaSuccess) {
        stage.buf = nullptr;
        cudaGetLastError();
        if (needed) return fail(CLAW_E_CUDA, "%s", cudaGetErrorString(e));
        return 0;
    }
    stage.n = n;
    return 0;
}

}  // namespace clawb200
