// Loan of the page-locked rings (see copy_ring.h).
#include "copy_ring.h"

#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

namespace pbs {

namespace {

constexpr int kVolumesPerRing = 32;

struct DeviceRings {
    std::vector<std::unique_ptr<CopyRing>> rings;
    int users = 0, volumes = 0;
};

// Never destroyed: contexts may go in static destructors.
struct Pools {
    std::mutex m;
    std::map<int, DeviceRings> devices;
};
Pools& pools() {
    static Pools* p = new Pools;
    return *p;
}

void free_ring(CopyRing& r) {
    for (cudaEvent_t e : r.done)
        if (e) cudaEventDestroy(e);
    if (r.mem) cudaFreeHost(r.mem);
}

std::unique_ptr<CopyRing> make_ring() {
    std::unique_ptr<CopyRing> r(new CopyRing);
    void* mem = nullptr;
    bool ok = cudaMallocHost(&mem, CopyRing::kSlots * CopyRing::kSlotBytes) == cudaSuccess;
    r->mem = ok ? static_cast<float*>(mem) : nullptr;
    for (cudaEvent_t& e : r->done) {
        if (ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            e = nullptr;
            ok = false;
        }
    }
    if (ok) return r;
    free_ring(*r);
    cudaGetLastError();
    return nullptr;
}

bool transfers_done(const CopyRing& r) {
    for (cudaEvent_t e : r.done) {
        if (cudaEventQuery(e) == cudaSuccess) continue;
        cudaGetLastError();
        return false;
    }
    return true;
}

}  // namespace

void CopyRingUser::begin(int device) {
    if (device_ >= 0) return;
    Pools& p = pools();
    std::lock_guard<std::mutex> lk(p.m);
    ++p.devices[device].users;
    device_ = device;
}

void CopyRingUser::end() {
    if (device_ < 0) return;
    Pools& p = pools();
    std::lock_guard<std::mutex> lk(p.m);
    DeviceRings& d = p.devices[device_];
    device_ = -1;
    if (--d.users > 0) return;
    for (auto& r : d.rings) free_ring(*r);
    d.rings.clear();
    d.volumes = 0;
}

CopyRingLoan::CopyRingLoan(int device, cudaStream_t s, bool volume) : stream_(s) {
    Pools& p = pools();
    std::lock_guard<std::mutex> lk(p.m);
    DeviceRings& d = p.devices[device];
    if (volume && d.volumes < kVolumesPerRing) ++d.volumes;
    for (auto& r : d.rings)
        if (!r->taken && transfers_done(*r)) ring_ = r.get();
    if (!ring_)
        for (auto& r : d.rings)
            if (!r->taken && r->last == s) ring_ = r.get();
    if (!ring_ && d.rings.size() < kMaxRings && (!volume || d.volumes >= kVolumesPerRing)) {
        try {
            d.rings.reserve(kMaxRings);
            if (std::unique_ptr<CopyRing> r = make_ring()) {
                ring_ = r.get();
                d.rings.push_back(std::move(r));
            }
        } catch (const std::exception&) {
        }
    }
    if (ring_) ring_->taken = true;
}

CopyRingLoan::~CopyRingLoan() {
    if (!ring_) return;
    std::lock_guard<std::mutex> lk(pools().m);
    ring_->last = stream_;
    ring_->taken = false;
}

}  // namespace pbs
