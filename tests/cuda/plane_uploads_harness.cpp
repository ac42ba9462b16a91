// Host-only harness: how planes at given addresses are gathered into copies
// (mmrecode_gb300/csrc/plane_uploads.h).
#include <stddef.h>
#include <stdint.h>

#include "plane_uploads.h"

// Planes [at[i], at[i] + size[i]), pinned ranges [lo[j], hi[j]). copy_of[i]: the number of the
// copy that plane i goes up with.
extern "C" void mmr_test_plane_uploads(const uint64_t *at, const uint64_t *size, size_t n, const uint64_t *lo,
                                       const uint64_t *hi, size_t n_ranges, uint32_t *copy_of) {
    auto ptr = [](uint64_t a) { return reinterpret_cast<const uint8_t *>(a); };
    auto range_of = [&](const uint8_t *p) {
        for (size_t j = 0; j < n_ranges; j++)
            if (p >= ptr(lo[j]) && p < ptr(hi[j])) return mmr::HostRange{ptr(lo[j]), ptr(hi[j])};
        return mmr::HostRange{};
    };
    mmr::PlaneUploads up;
    uint32_t copies = 0;
    for (size_t i = 0; i < n; i++) {
        if (!up.append(ptr(at[i]), size[i], range_of)) {
            up.start(ptr(at[i]), nullptr, size[i], range_of);
            copies++;
        }
        copy_of[i] = copies - 1;
    }
}
