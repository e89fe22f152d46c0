// Copies between pageable host memory and the device for the host-buffer entry points.
//
// A pageable cudaMemcpy runs through the driver's own staging on one thread: 5 GB/s down, and
// every page of a fresh NumPy buffer is faulted in on that thread (a 500 x 389 far block: 7.8
// ms down, 2 ms up for 37 MB, the kernel 0.44 ms).  Here a few threads copy 1 MiB chunks
// through pinned slots of the handle, each chunk's PCIe transfer under the other threads'
// memory copies and page faults.  The slots (16 MiB) are the handle's, allocated at the first
// large copy and given back with its workspaces; the threads live for one call.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

#include "common.cuh"

#define STAGE_CHUNK ((size_t)1 << 20)
#define STAGE_THREADS 8
#define STAGE_SLOTS (2 * STAGE_THREADS)
// From these totals on the threads cost less than the plain copy: up, from buffers that are in
// place (64 x 2000, 2.1 MB 0.89 ms plain, 0.95 staged; 300 x 300, 2.9 MB 1.50, 1.54; 450 x 181, 4.5
// MB 1.96, 1.83; 900 x 1, 13 MB 3.56, 3.02), and down, into fresh pages (far blocks of 1.9 MB 0.52,
// 0.48; 3.1 MB 0.73, 0.56; 12.6 MB 2.07, 1.02).
#define STAGE_MIN_UP ((size_t)4 << 20)
#define STAGE_MIN_DOWN ((size_t)2 << 20)

struct HostCopy {
    void *device, *host;
    size_t bytes;
};

static void stage_free(grim_context *h) {
    for (size_t i = 0; i < h->stage_events.size(); ++i) {
        if (h->stage_pending[i]) cudaEventSynchronize(h->stage_events[i]);
        cudaEventDestroy(h->stage_events[i]);
    }
    h->stage_events.clear();
    h->stage_pending.clear();
    if (h->stage) cudaFreeHost(h->stage);
    h->stage = nullptr;
}

static bool stage_ready(grim_context *h) {
    if (h->stage) return true;
    if (cudaHostAlloc(&h->stage, STAGE_SLOTS * STAGE_CHUNK, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();  // no pinned memory left: the plain copies
        h->stage = nullptr;
        return false;
    }
    for (int i = 0; i < STAGE_SLOTS; ++i) {
        cudaEvent_t e;
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            stage_free(h);
            return false;
        }
        h->stage_events.push_back(e);
        h->stage_pending.push_back(0);
    }
    return true;
}

// The copies of `list`, in stream order on the handle's stream, up (host to device; the host
// buffers are read in stream order at the latest) or down (returns when they have been written).  On
// cudaStreamPerThread, which names another stream on every thread, the plain copies.
static int stage_copy(grim_context *h, const std::vector<HostCopy> &list, bool up) {
    size_t total = 0;
    for (const HostCopy &c : list) total += c.bytes;
    const cudaMemcpyKind kind = up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    if (total < (up ? STAGE_MIN_UP : STAGE_MIN_DOWN) || h->stream == cudaStreamPerThread || !stage_ready(h)) {
        for (const HostCopy &c : list)
            GRIM_CHECK_CUDA(cudaMemcpyAsync(up ? c.device : c.host, up ? c.host : c.device, c.bytes, kind, h->stream));
        if (!up) GRIM_CHECK_CUDA(cudaStreamSynchronize(h->stream));
        return GRIM_OK;
    }
    std::vector<HostCopy> chunks;
    for (const HostCopy &c : list)
        for (size_t at = 0; at < c.bytes; at += STAGE_CHUNK)
            chunks.push_back({(char *)c.device + at, (char *)c.host + at, std::min(STAGE_CHUNK, c.bytes - at)});
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency() / 2);
    const int threads = (int)std::min<size_t>({(size_t)STAGE_THREADS, (size_t)cores, chunks.size()});
    std::atomic<int> error{(int)cudaSuccess};
    const cudaStream_t stream = h->stream;
    // thread t: chunks t, t + threads, ... through its own two slots
    auto work = [&, threads, up](int t) {
        cudaError_t e = cudaSetDevice(h->device);
        int pending[2] = {-1, -1};  // chunk in flight in a slot (down: still to be copied out)
        auto finish = [&](int s) {
            const int slot = 2 * t + s;
            if (e == cudaSuccess && h->stage_pending[slot]) e = cudaEventSynchronize(h->stage_events[slot]);
            h->stage_pending[slot] = 0;
            if (!up && e == cudaSuccess && pending[s] >= 0)
                std::memcpy(chunks[pending[s]].host, (char *)h->stage + slot * STAGE_CHUNK, chunks[pending[s]].bytes);
            pending[s] = -1;
        };
        int s = 0;
        for (size_t c = t; c < chunks.size() && e == cudaSuccess; c += threads, s ^= 1) {
            finish(s);
            if (e != cudaSuccess) break;
            const int slot = 2 * t + s;
            char *pin = (char *)h->stage + slot * STAGE_CHUNK;
            if (up) std::memcpy(pin, chunks[c].host, chunks[c].bytes);
            e = cudaMemcpyAsync(up ? chunks[c].device : pin, up ? pin : chunks[c].device, chunks[c].bytes, kind, stream);
            if (e == cudaSuccess) e = cudaEventRecord(h->stage_events[slot], stream);
            if (e != cudaSuccess) break;
            h->stage_pending[slot] = 1;
            pending[s] = (int)c;
        }
        if (!up)
            for (int i = 0; i < 2; ++i, s ^= 1) finish(s);
        if (e != cudaSuccess) error = (int)e;
    };
    std::vector<std::thread> team;
    int started = 1;
    try {
        team.reserve(threads);
        for (; started < threads; ++started) team.emplace_back(work, started);
    } catch (const std::exception &) {
        // no thread to be had: the calling thread takes their chunks too
    }
    work(0);
    for (int t = started; t < threads; ++t) work(t);
    for (std::thread &t : team) t.join();
    if (error != (int)cudaSuccess) return grim_cuda_check((cudaError_t)error.load(), "host copy");
    return GRIM_OK;
}

// dst[c][r] = src[r][c] (rows x cols, row-major, to column-major leading dimension ldd); the grid
// covers the columns, its y extent steps over the rows.
__global__ void k_transpose(int rows, int cols, const double2 *__restrict__ src, int64_t lds, double2 *__restrict__ dst,
                            int64_t ldd) {
    __shared__ double2 tile[32][33];
    const int c0 = blockIdx.x * 32;
    for (int64_t r0 = (int64_t)blockIdx.y * 32; r0 < rows; r0 += (int64_t)gridDim.y * 32) {
        for (int i = threadIdx.y; i < 32; i += blockDim.y)
            if (r0 + i < rows && c0 + threadIdx.x < cols) tile[i][threadIdx.x] = src[(r0 + i) * lds + c0 + threadIdx.x];
        __syncthreads();
        for (int i = threadIdx.y; i < 32; i += blockDim.y)
            if (c0 + i < cols && r0 + threadIdx.x < rows)
                dst[(int64_t)(c0 + i) * ldd + r0 + threadIdx.x] = tile[threadIdx.x][i];
        __syncthreads();
    }
}
