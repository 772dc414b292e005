// Host <-> device transfers of the drop-in calls (mdg_force_get, mdg_shake).
//
// Pinned host memory is mapped into the GPU's address space; on a Grace-Blackwell node the GPU
// reaches it over the coherent NVLink-C2C link.  A call moves a dozen or more separate arrays
// (positions, offsets, centres in; forces, torques, energies, status out), and one DMA copy per
// array costs a few microseconds of setup latency each, serialised on the stream.  Here every
// array whose host side is pinned joins one batch that a single kernel copies (one CTA column per
// array, 8-byte words, so the bits move unchanged); the others go through cudaMemcpyAsync.

#include <mutex>

#include "ctx.h"
#include "pinned.h"

namespace mdg {

namespace {

// Ranges pinned through mdg_pin_host.  They stay valid until mdg_unpin_host, so a call finds its arrays here without
// asking the driver.
std::mutex g_pin_mu;
PinnedRanges g_pinned;

__global__ void k_io_copy(IoBatch b) {
    const int s = blockIdx.y;
    const unsigned long long* __restrict__ src = b.src[s];
    unsigned long long* __restrict__ dst = b.dst[s];
    const long n = b.n[s];
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

// The GPU's address of an array in host memory that CUDA knows as pinned, or nullptr.
void* pinned_address(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();  // some drivers report memory CUDA does not know as an error: clear it
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost ? a.devicePointer : nullptr;
}

// The GPU's address of a host array and into `room` how many of its bytes it reaches from there: all of them, but for
// an array that runs over the end of a range given to mdg_pin_host.  nullptr (and 0) when the array is not pinned, at
// its end as at its start: pageable memory is copied through the driver's staging instead.
void* mapped_address(const void* p, size_t bytes, size_t& room) {
    {
        std::lock_guard<std::mutex> lk(g_pin_mu);
        if (void* r = g_pinned.find(p, bytes, room)) return r;
    }
    char* first = static_cast<char*>(pinned_address(p));
    if (!first || pinned_address(static_cast<const char*>(p) + bytes - 1) != first + bytes - 1) return nullptr;
    room = bytes;
    return first;
}

}  // namespace

cudaError_t io_add(Ctx& c, IoBatch& b, void* dst, const void* src, long nwords, bool h2d) {
    if (nwords <= 0 || !dst || !src) return cudaSuccess;
    const cudaMemcpyKind kind = h2d ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    size_t bytes = sizeof(unsigned long long) * nwords, room = 0;
    void* m = b.nseg < IoBatch::kMax ? mapped_address(h2d ? src : dst, bytes, room) : nullptr;
    char* d = static_cast<char*>(dst);
    const char* h = static_cast<const char*>(src);
    if (room >= sizeof(unsigned long long)) {
        b.src[b.nseg] = static_cast<const unsigned long long*>(h2d ? m : src);
        b.dst[b.nseg] = static_cast<unsigned long long*>(h2d ? dst : m);
        b.n[b.nseg] = (long)(room / 8);
        b.nmax = std::max(b.nmax, b.n[b.nseg]);
        ++b.nseg;
    }
    // what the kernel does not take: a word that the pinned range ends in, the rest beyond it, or all of a pageable array
    const size_t words = room / 8 * 8;
    for (size_t at = words; at < bytes;) {
        const size_t n = at < room ? room - at : bytes - at;
        const cudaError_t e = cudaMemcpyAsync(d + at, h + at, n, kind, c.stream);
        if (e != cudaSuccess) return e;
        at += n;
    }
    return cudaSuccess;
}

void io_add_device(IoBatch& b, void* dst, const void* src, long nwords) {
    b.src[b.nseg] = static_cast<const unsigned long long*>(src);
    b.dst[b.nseg] = static_cast<unsigned long long*>(dst);
    b.n[b.nseg] = nwords;
    b.nmax = std::max(b.nmax, nwords);
    ++b.nseg;
}

cudaError_t pin_host_range(void* p, size_t bytes) {
    cudaError_t e = cudaHostRegister(p, bytes, cudaHostRegisterMapped | cudaHostRegisterPortable);
    if (e != cudaSuccess) return e;
    void* d = nullptr;
    e = cudaHostGetDevicePointer(&d, p, 0);
    if (e != cudaSuccess) {
        cudaHostUnregister(p);
        return e;
    }
    std::lock_guard<std::mutex> lk(g_pin_mu);
    g_pinned.add(p, bytes, d);
    return cudaSuccess;
}

cudaError_t unpin_host_range(void* p) {
    {
        std::lock_guard<std::mutex> lk(g_pin_mu);
        g_pinned.remove(p);
    }
    return cudaHostUnregister(p);
}

void io_flush(Ctx& c, IoBatch& b) {
    if (b.nseg == 0) return;
    const int gx = (int)std::min<long>((b.nmax + 255) / 256, 32);
    k_io_copy<<<dim3(gx, b.nseg), 256, 0, c.stream>>>(b);
    b.nseg = 0;
    b.nmax = 0;
}

}  // namespace mdg
