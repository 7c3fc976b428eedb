// context.cpp - which CUDA context device memory belongs to.
//
// A cudaDeviceReset destroys a device's context with all its memory and modules;
// the next call makes a new one, which the driver hands out under the same
// pointer.  What tells the two apart is cuCtxGetId, unique for the life of the
// process.  The driver's functions come from the runtime's entry point table, as
// the library does not link libcuda, so that it loads on machines without a GPU.
#include "internal.hpp"

namespace mcg {
namespace {

using Context = void *;
template <class F>
F driver_entry(const char *name) {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return reinterpret_cast<F>(f);
}

uint64_t id_of(Context ctx) {
    static const auto get_id = driver_entry<int (*)(Context, unsigned long long *)>("cuCtxGetId");
    unsigned long long id = 0;
    return ctx && get_id && get_id(ctx, &id) == 0 ? uint64_t(id) : 0;
}

Context current_context() {
    static const auto get_current = driver_entry<int (*)(Context *)>("cuCtxGetCurrent");
    Context ctx = nullptr;
    return get_current && get_current(&ctx) == 0 ? ctx : nullptr;
}

// Null while it is not active; asking does not activate it.
Context primary_context(int device) {
    static const auto get_state = driver_entry<int (*)(int, unsigned *, int *)>("cuDevicePrimaryCtxGetState");
    static const auto retain = driver_entry<int (*)(Context *, int)>("cuDevicePrimaryCtxRetain");
    static const auto release = driver_entry<int (*)(int)>("cuDevicePrimaryCtxRelease");
    unsigned flags = 0;
    int active = 0;
    Context ctx = nullptr;
    if (!get_state || !retain || !release || get_state(device, &flags, &active) != 0 || !active) return nullptr;
    if (retain(&ctx, device) != 0) return nullptr;
    release(device);
    return ctx;
}

}  // namespace

uint64_t current_context_id() { return id_of(current_context()); }

uint64_t primary_context_id(int device) { return id_of(primary_context(device)); }

}  // namespace mcg
