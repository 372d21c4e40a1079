// Which shared-memory limits of kernels are set. No CUDA in here: itb_ctx.cu binds it to the runtime (itb_raise_smem).
#pragma once
#include <stddef.h>

#include <mutex>
#include <unordered_map>

// A kernel's limit is kept per device, and every context and thread of the process shares it: setting it for one device leaves the
// others at 48 KB, and setting it to what one caller needs lowers it for another that needs more. So one table for the process, by
// device, that only ever raises.
class SmemLimits {
    static constexpr int N_DEV = 64;
    std::mutex mu;
    std::unordered_map<const void*, size_t> have[N_DEV];

public:
    // Makes `fn` launchable with `bytes` of dynamic shared memory on `device`. set() applies the limit there and returns 0, or an error,
    // which is handed back and leaves the table as it was.
    template <class Set>
    auto raise(int device, const void* fn, size_t bytes, Set&& set) -> decltype(set()) {
        if (device < 0 || device >= N_DEV) return set();
        std::lock_guard<std::mutex> hold(mu);
        size_t& h = have[device][fn];
        if (bytes <= h) return {};
        const auto e = set();
        if (e == decltype(e){}) h = bytes;
        return e;
    }
};
