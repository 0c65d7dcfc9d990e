// Device blocks kept between owners.
//
// Building or dropping a matrix takes ~20 allocations, each ~130 us in
// cudaMalloc and again in cudaFree: 5.8 of the 9 ms of a Galerkin product of a
// 263 k-row matrix.  A released block is kept, by device and size class, and
// handed to the next allocation of that class.
//   * Safety: a block may be handed out once no queued work uses it any more.  All
//     work of the library runs on its contexts' streams (what a batched call runs
//     beside it is joined before the call returns), so a release waits for these,
//     1.5 us a context when they are idle.  It does not wait for the device: that
//     is an error, and breaks the capture, while any stream of the device is being
//     captured, whoever's it is.  While a solver of this process captures
//     (CaptureScope), or one of these streams is found capturing, the release is a
//     plain cudaFree, which other threads may call during a thread-local capture.
//   * Bound: at most kPoolCap bytes per device are kept, in blocks of at most
//     kPoolBlock (larger ones are freed at once); beyond that the block kept for
//     longest goes, or a pool filled by other sizes would keep nothing any more.
//     pool_trim gives everything back (jfg_release_scratch, jfg_destroy, and before
//     an allocation that the device refuses is tried again).
#include <algorithm>
#include <list>
#include <map>
#include <mutex>

#include "jfg_common.cuh"

namespace jfg {
namespace {

constexpr size_t kPoolCap = (size_t)1 << 30;
constexpr size_t kPoolBlock = (size_t)256 << 20;

struct Block {
    size_t c;                                      // class
    void* p;
};
struct Kept {                                      // the free blocks of a device
    std::list<Block> all;                          // oldest first
    std::map<size_t, std::vector<std::list<Block>::iterator>> of;   // by class, oldest first
    size_t bytes = 0;

    void* take(size_t c)                           // the newest of a class
    {
        auto f = of.find(c);
        if (f == of.end() || f->second.empty()) return nullptr;
        auto b = f->second.back();
        f->second.pop_back();
        void* p = b->p;
        all.erase(b);
        bytes -= c;
        return p;
    }
    void put(size_t c, void* p)
    {
        auto& v = of[c];
        v.reserve(v.size() + 1);                   // nothing throws after the block is in the list
        all.push_back(Block{c, p});
        v.push_back(std::prev(all.end()));
        bytes += c;
    }
    void* drop_oldest()
    {
        const Block b = all.front();
        auto& v = of[b.c];
        v.erase(v.begin());
        all.pop_front();
        bytes -= b.c;
        return b.p;
    }
};
struct Pool {
    std::mutex m;
    std::map<int, Kept> of;
};
Pool& pool()
{
    static Pool* p = new Pool();      // never destroyed: buffers of static objects outlive it otherwise
    return *p;
}

struct Streams {
    std::mutex m;                                  // held while streams are waited for: no capture begins then
    int capturing = 0;
    std::map<int, std::vector<cudaStream_t>> of;   // the library's streams by device
};
Streams& streams()
{
    static Streams* s = new Streams();
    return *s;
}

// Waits for the library's streams of a device; false when it may not or cannot.
bool wait_streams(int dev)
{
    Streams& S = streams();
    std::lock_guard<std::mutex> g(S.m);
    if (S.capturing) return false;
    for (cudaStream_t st : S.of[dev]) {
        cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &c) != cudaSuccess || c != cudaStreamCaptureStatusNone ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            cudaGetLastError();                    // not the caller's: its next launch check may not find it
            return false;
        }
    }
    return true;
}

// Eight classes per power of two, multiples of 512 bytes, up to steps of 2 MB (the
// granularity of cudaMalloc, so a large block is no larger than it would be there).
size_t size_class(size_t bytes)
{
    size_t step = 512;
    while (step * 16 <= bytes && step < ((size_t)2 << 20)) step *= 2;
    return (bytes + step - 1) / step * step;
}

struct DeviceGuard {
    int old = -1, dev;
    explicit DeviceGuard(int d) : dev(d)
    {
        if (cudaGetDevice(&old) == cudaSuccess && old != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard()
    {
        if (old >= 0 && old != dev) cudaSetDevice(old);
    }
};

}  // namespace

void* pool_alloc(size_t bytes, int* dev)
{
    JFG_CUDA(cudaGetDevice(dev));
    const size_t c = size_class(bytes);
    Pool& p = pool();
    if (c <= kPoolBlock) {
        std::lock_guard<std::mutex> g(p.m);
        if (void* b = p.of[*dev].take(c)) return b;
    }
    const size_t size = c <= kPoolBlock ? c : bytes;      // a block that is never kept is not rounded up
    void* b = nullptr;
    cudaError_t e = cudaMalloc(&b, size);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        pool_trim(*dev);
        e = cudaMalloc(&b, size);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw Error{JFG_ERR_CUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e)};
    }
    return b;
}

void pool_free(void* b, size_t bytes, int dev) noexcept
{
    const size_t c = size_class(bytes);
    DeviceGuard on(dev);
    Pool& p = pool();
    if (c <= kPoolBlock) {
        try {
            if (wait_streams(dev)) {
                std::vector<void*> old;
                {
                    std::lock_guard<std::mutex> g(p.m);
                    Kept& k = p.of[dev];
                    old.reserve(k.all.size());
                    k.put(c, b);
                    while (k.bytes > kPoolCap) old.push_back(k.drop_oldest());
                }
                for (void* o : old) cudaFree(o);
                return;
            }
        } catch (...) {
        }
    }
    cudaFree(b);
}

void pool_add_stream(int dev, cudaStream_t st)
{
    Streams& S = streams();
    std::lock_guard<std::mutex> g(S.m);
    S.of[dev].push_back(st);
}

void pool_drop_stream(int dev, cudaStream_t st) noexcept
{
    Streams& S = streams();
    std::lock_guard<std::mutex> g(S.m);
    auto it = S.of.find(dev);
    if (it == S.of.end()) return;
    auto& v = it->second;
    v.erase(std::remove(v.begin(), v.end(), st), v.end());
}

CaptureScope::CaptureScope()
{
    std::lock_guard<std::mutex> g(streams().m);
    streams().capturing++;
}

CaptureScope::~CaptureScope()
{
    std::lock_guard<std::mutex> g(streams().m);
    streams().capturing--;
}

void pool_trim(int dev) noexcept
{
    DeviceGuard on(dev);
    Pool& p = pool();
    std::lock_guard<std::mutex> g(p.m);
    Kept& k = p.of[dev];
    while (!k.all.empty()) cudaFree(k.drop_oldest());
}

}  // namespace jfg
