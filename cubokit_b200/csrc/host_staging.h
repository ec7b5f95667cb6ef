// Host staging memory for the object and probe transfers, grown on demand and kept: page-locked (copies run at full link speed
// and its pages are already mapped) or, where the driver has none left, pageable.
#pragma once

#include <cstddef>
#include <cstdint>
#include <memory>

namespace cubo {

class HostStaging {
  public:
    // allocate returns null where it cannot
    HostStaging(void *(*allocate)(size_t), void (*free)(void *)) : allocate_(allocate), free_(free) {}
    HostStaging(const HostStaging &) = delete;
    HostStaging &operator=(const HostStaging &) = delete;
    ~HostStaging() { release(); }
    // At least `bytes`, aligned for any type; the contents are not kept when it grows.  Throws std::bad_alloc.
    void *get(size_t bytes) {
        if (bytes_ >= bytes) return pinned_ ? pinned_ : pageable_.get();
        release();
        pinned_ = allocate_(bytes);
        if (!pinned_) pageable_.reset(new uint8_t[bytes]);
        bytes_ = bytes;
        return pinned_ ? pinned_ : pageable_.get();
    }

  private:
    void release() {
        if (pinned_) free_(pinned_);
        pinned_ = nullptr;
        pageable_.reset();
        bytes_ = 0;
    }
    void *(*allocate_)(size_t);
    void (*free_)(void *);
    void *pinned_ = nullptr;
    std::unique_ptr<uint8_t[]> pageable_;
    size_t bytes_ = 0;
};

// One staged transfer of `probe_values` complex128 values, the object (or its gradient) in the plan's type and one double:
// every transfer of a plan has the same size, so the first one's memory serves them all.
struct StagedState {
    uint8_t *probe, *object;
    double *value;
    StagedState(HostStaging &staging, size_t probe_values, size_t object_bytes) {
        const size_t probe_bytes = probe_values * 2 * sizeof(double);
        probe = static_cast<uint8_t *>(staging.get(probe_bytes + object_bytes + sizeof(double)));
        object = probe + probe_bytes;
        value = reinterpret_cast<double *>(object + object_bytes);
    }
};

}  // namespace cubo
