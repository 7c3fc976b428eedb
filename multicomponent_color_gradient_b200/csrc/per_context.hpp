// per_context.hpp - one shared object per device and CUDA context.
#pragma once

#include <cstdint>
#include <map>
#include <memory>
#include <mutex>

namespace mcg {

// Objects made as T(device, context) that live while someone holds them.
// `context` identifies a device's context for the life of the process
// (current_context_id): after a cudaDeviceReset the next holder gets a new
// object, and those of the old context keep theirs.
template <class T>
class PerContext {
public:
    std::shared_ptr<T> get(int device, uint64_t context) {
        std::lock_guard<std::mutex> lock(m_);
        Known &k = known_[device];
        std::shared_ptr<T> s = k.context == context ? k.object.lock() : nullptr;
        if (!s) {
            s = std::make_shared<T>(device, context);
            k.context = context;
            k.object = s;
        }
        return s;
    }

private:
    struct Known {
        uint64_t context = 0;
        std::weak_ptr<T> object;
    };
    std::mutex m_;
    std::map<int, Known> known_;
};

}  // namespace mcg
