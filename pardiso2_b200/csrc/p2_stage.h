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
    // The slots are made (3 to 4 ms of page-locking) with the heat rows of a grid of
    // at least kLikelyNodes nodes, on a smaller one when a list of at least kLeast
    // pageable bytes arrives; from then on every list goes through them.  Heat steps
    // with / without: fields and markers of 3 + 4 MB 5.56 / 5.52 ms, 6 + 9 MB 5.84 /
    // 5.88, 10 + 15 MB 5.76 / 6.10, 23 + 4 MB 5.39 / 5.92, 23 + 36 MB 6.9 / 9.4: a small
    // step would not earn them.
    static constexpr long kLikelyNodes = 50000;
    static constexpr size_t kLeast = 40 * kPiece;

    ~HostStage()
    {
        for (cudaEvent_t e : ev)
            if (e) {
                cudaEventSynchronize(e);
                cudaEventDestroy(e);
            }
        if (buf) cudaFreeHost(buf);
    }
    // The slots and their events; false when the host gives no page-locked memory.
    bool reserve()
    {
        if (buf) return true;
        const unsigned hw = std::thread::hardware_concurrency();
        workers = (int)std::min<unsigned>(kWorkers, std::max(1u, hw / 2));
        ev.resize((size_t)workers * kSlots, nullptr);
        for (cudaEvent_t &e : ev)
            if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                e = nullptr;
                cudaGetLastError();
                return false;
            }
        if (cudaMallocHost((void **)&buf, kPiece * workers * kSlots) != cudaSuccess) {
            buf = nullptr;
            cudaGetLastError();
            return false;
        }
        return true;
    }

    // Issues the copies on the stream: page-locked arrays directly, others in
    // pieces (directly while there are no slots).  To the device: returns once the pageable
    // arrays have been read.  To the host: once they have been written.
    cudaError_t run(int device, std::vector<HostCopy> list, cudaMemcpyKind kind, cudaStream_t st)
    {
        const bool up = kind == cudaMemcpyHostToDevice;
        struct Piece { char *dev, *host; size_t bytes; };
        std::vector<Piece> pieces;
        size_t total = 0;
        std::vector<char> pageable(list.size());
        for (size_t q = 0; q < list.size(); q++) {
            cudaPointerAttributes at{};
            if (cudaPointerGetAttributes(&at, list[q].host) != cudaSuccess) cudaGetLastError();
            pageable[q] = !(at.type == cudaMemoryTypeHost || at.type == cudaMemoryTypeManaged || at.type == cudaMemoryTypeDevice);
            if (pageable[q]) total += list[q].bytes;
        }
        const bool staged = buf || (total >= kLeast && reserve());
        for (size_t q = 0; q < list.size(); q++) {
            const HostCopy &c = list[q];
            if (!pageable[q] || !staged) {
                const cudaError_t e = up ? cudaMemcpyAsync(c.dev, c.host, c.bytes, kind, st)
                                         : cudaMemcpyAsync(c.host, c.dev, c.bytes, kind, st);
                if (e != cudaSuccess) return e;
                continue;
            }
            for (size_t o = 0; o < c.bytes; o += kPiece)
                pieces.push_back(Piece{(char *)c.dev + o, (char *)c.host + o, std::min(kPiece, c.bytes - o)});
        }
        if (pieces.empty()) return cudaSuccess;
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
