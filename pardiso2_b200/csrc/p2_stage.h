// Copies between pageable host arrays and the device.
//
// A copy of pageable memory by the runtime is filled by one thread at about
// 10 GB/s, and copies issued by several threads wait for one another: the 68 MB
// of fields and markers of a heat step on 65^3 nodes bound it.  Here up to four
// threads copy pieces through page-locked slots of their own, so that several
// are in flight: that step 8.4 -> 6.7 ms between its events, 9.7 -> 8.0 ms as
// called.  Page-locked arrays are copied directly.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <thread>
#include <vector>

#include "p2_internal.cuh"

namespace p2 {

struct HostCopy {
    void *dev, *host;
    size_t bytes;
};

// One transfer at a time; a context owns one.
class HostStage {
  public:
    static constexpr size_t kPiece = (size_t)256 << 10;
    static constexpr int kWorkers = 4, kSlots = 3;

    ~HostStage()
    {
        for (cudaEvent_t e : ev)
            if (e) {
                cudaEventSynchronize(e);
                cudaEventDestroy(e);
            }
        if (buf) cudaFreeHost(buf);
    }
    void reserve()
    {
        if (buf) return;
        const unsigned hw = std::thread::hardware_concurrency();
        workers = (int)std::min<unsigned>(kWorkers, std::max(1u, hw / 2));
        ev.assign((size_t)workers * kSlots, nullptr);
        for (cudaEvent_t &e : ev) P2_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        P2_CUDA_TRY(cudaMallocHost((void **)&buf, kPiece * workers * kSlots));
    }
    // Issues the copies on the stream: page-locked arrays directly, others in
    // pieces.  To the device: returns once the pageable arrays have been read.
    // To the host: once they have been written.
    cudaError_t run(int device, std::vector<HostCopy> list, cudaMemcpyKind kind, cudaStream_t st)
    {
        const bool up = kind == cudaMemcpyHostToDevice;
        struct Piece { char *dev, *host; size_t bytes; };
        std::vector<Piece> pieces;
        for (const HostCopy &c : list) {
            cudaPointerAttributes at{};
            if (cudaPointerGetAttributes(&at, c.host) != cudaSuccess) cudaGetLastError();
            if (at.type == cudaMemoryTypeHost || at.type == cudaMemoryTypeManaged || at.type == cudaMemoryTypeDevice) {
                const cudaError_t e = up ? cudaMemcpyAsync(c.dev, c.host, c.bytes, kind, st)
                                         : cudaMemcpyAsync(c.host, c.dev, c.bytes, kind, st);
                if (e != cudaSuccess) return e;
                continue;
            }
            for (size_t o = 0; o < c.bytes; o += kPiece)
                pieces.push_back(Piece{(char *)c.dev + o, (char *)c.host + o, std::min(kPiece, c.bytes - o)});
        }
        std::atomic<size_t> next{0};
        std::atomic<int> error{(int)cudaSuccess};
        auto work = [&](int w) {
            cudaError_t e = cudaSetDevice(device);
            Piece held[kSlots] = {};  // to the host: pieces in flight, by slot
            bool busy[kSlots] = {};
            char *slot0 = buf + kPiece * kSlots * w;
            auto land = [&](int q) {  // a piece that has arrived in its slot
                if (!busy[q]) return;
                busy[q] = false;
                if (e == cudaSuccess) e = cudaEventSynchronize(ev[w * kSlots + q]);
                if (e == cudaSuccess) std::memcpy(held[q].host, slot0 + kPiece * q, held[q].bytes);
            };
            int q = 0;
            for (; e == cudaSuccess && error.load() == (int)cudaSuccess; q = (q + 1) % kSlots) {
                const size_t i = next.fetch_add(1);
                if (i >= pieces.size()) break;
                const Piece &P = pieces[i];
                char *s = slot0 + kPiece * q;
                if (up) {
                    e = cudaEventSynchronize(ev[w * kSlots + q]);
                    if (e == cudaSuccess) {
                        std::memcpy(s, P.host, P.bytes);
                        e = cudaMemcpyAsync(P.dev, s, P.bytes, kind, st);
                    }
                } else {
                    land(q);
                    if (e == cudaSuccess) e = cudaMemcpyAsync(s, P.dev, P.bytes, kind, st);
                    held[q] = P;
                    busy[q] = e == cudaSuccess;
                }
                if (e == cudaSuccess) e = cudaEventRecord(ev[w * kSlots + q], st);
            }
            for (int k = 0; k < kSlots; k++) land((q + k) % kSlots);
            if (e != cudaSuccess) error.store((int)e);
        };
        const int n = (int)std::min<size_t>(workers, pieces.size() / 4);
        std::vector<std::thread> th;
        for (int w = 1; w < n; w++) {
            try {
                th.emplace_back(work, w);
            } catch (...) {  // no more threads: the rest is this one's
                break;
            }
        }
        work(0);
        for (auto &t : th) t.join();
        return (cudaError_t)error.load();
    }

  private:
    char *buf = nullptr;
    int workers = 1;
    std::vector<cudaEvent_t> ev;
};

}  // namespace p2
