// Copies between pageable host memory and the device.
//
// The driver copies pageable memory through a pinned buffer of its own with one
// thread, about 10 GB/s, and the call returns only when the copy is done, so nothing
// else is queued meanwhile.  Here several threads each move pieces through two pinned
// slots: the memory copy (and the page faults of a fresh result) run in parallel and
// overlap the transfers.
#include "internal.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <new>
#include <thread>
#include <vector>

namespace ctlcu {

cudaError_t HostCopier::ensure()
{
    if (ready)
        return cudaSuccess;
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    workers = (int)std::min<unsigned>(kMaxWorkers, std::max(1u, hw / 2));
    cudaError_t e = cudaHostAlloc(&base, kSlot * 2 * workers, cudaHostAllocDefault);
    for (int i = 0; e == cudaSuccess && i < 2 * workers; ++i)
        e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
    if (e != cudaSuccess) {
        release();
        cudaGetLastError();
        return e;
    }
    ready = true;
    return cudaSuccess;
}

void HostCopier::release()
{
    for (cudaEvent_t& x : ev) {
        if (x)
            cudaEventDestroy(x);
        x = nullptr;
    }
    if (base)
        cudaFreeHost(base);
    base = nullptr;
    ready = false;
}

namespace {

struct Piece {
    char* device;
    char* host;
    size_t bytes;
    cudaEvent_t after;  // to wait for, or null
};

std::vector<Piece> cut(const HostCopyPart* parts, size_t n)
{
    std::vector<Piece> out;
    for (size_t i = 0; i < n; ++i) {
        const HostCopyPart& p = parts[i];
        for (size_t o = 0; o < p.bytes; o += HostCopier::kSlot)
            out.push_back({ (char*)p.device + o, (char*)p.host + o, std::min(HostCopier::kSlot, p.bytes - o), p.after });
    }
    return out;
}

// Worker w of a copy: takes pieces in order, two in flight through its own two slots.
cudaError_t work(HostCopier& hc, int device, const std::vector<Piece>& pieces, std::atomic<size_t>& next, int w,
                 bool to_host, cudaStream_t st)
{
    cudaError_t e = cudaSetDevice(device);
    const Piece* in_flight[2] = { nullptr, nullptr };
    // a slot's transfer is over; towards the host its bytes then go to their place
    auto finish = [&](int s) {
        if (!in_flight[s])
            return;
        const cudaError_t r = cudaEventSynchronize(hc.ev[2 * w + s]);
        if (e == cudaSuccess)
            e = r;
        if (e == cudaSuccess && to_host)
            std::memcpy(in_flight[s]->host, hc.slot(2 * w + s), in_flight[s]->bytes);
        in_flight[s] = nullptr;
    };
    for (int s = 0; e == cudaSuccess; s ^= 1) {
        const size_t i = next.fetch_add(1);
        if (i >= pieces.size())
            break;
        const Piece& p = pieces[i];
        finish(s);
        if (e != cudaSuccess)
            break;
        char* slot = hc.slot(2 * w + s);
        if (to_host) {
            if (p.after)
                e = cudaStreamWaitEvent(st, p.after, 0);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(slot, p.device, p.bytes, cudaMemcpyDeviceToHost, st);
        } else {
            std::memcpy(slot, p.host, p.bytes);
            e = cudaMemcpyAsync(p.device, slot, p.bytes, cudaMemcpyHostToDevice, st);
        }
        if (e == cudaSuccess)
            e = cudaEventRecord(hc.ev[2 * w + s], st);
        if (e == cudaSuccess)
            in_flight[s] = &p;
    }
    // older first, so that pieces reach the host in order
    for (int s = 0; s < 2; ++s)
        finish(s);
    return e;
}

}  // namespace

// Returns when every byte is in place (to the host) or has left the slots (to the
// device: the transfers are queued on `st` and done).  No exception leaves it: it runs
// behind a C interface.
cudaError_t HostCopier::run(int device, const HostCopyPart* parts, size_t n_parts, bool to_host, cudaStream_t st)
try {
    const std::vector<Piece> pieces = cut(parts, n_parts);
    const int n = (int)std::min<size_t>((size_t)workers, pieces.size());
    std::atomic<size_t> next{ 0 };
    std::vector<cudaError_t> got((size_t)std::max(n, 1), cudaSuccess);
    std::vector<std::thread> threads;
    threads.reserve((size_t)std::max(n, 1));
    for (int w = 1; w < n; ++w) {
        try {
            threads.emplace_back([&, w] { got[(size_t)w] = work(*this, device, pieces, next, w, to_host, st); });
        } catch (const std::exception&) {
            break;  // no thread, or no memory for one: the threads there are take the pieces
        }
    }
    if (n > 0)
        got[0] = work(*this, device, pieces, next, 0, to_host, st);
    for (std::thread& t : threads)
        t.join();
    for (cudaError_t e : got)
        if (e != cudaSuccess)
            return e;
    return cudaSuccess;
} catch (const std::bad_alloc&) {
    return cudaErrorMemoryAllocation;  // before any thread was started
}

}  // namespace ctlcu
