// csrc/host_page.h with CUDA calls that can fail.  Bits of `fail`: 1 registering, 2 the device
// pointer, 4 a device pointer that is null.  out = {opened, opened again, registrations,
// releases, errors cleared, host left, dev left}.
#include "host_page.h"

namespace {
int g_fail, g_reg, g_unreg, g_clear;
struct Api {
    static bool register_page(void*, size_t n) {
        if (g_fail & 1) return false;
        ++g_reg;
        return n == eup::kHostPage;
    }
    static bool device_pointer(void* p, void** d) {
        *d = (g_fail & 4) ? nullptr : p;
        return !(g_fail & 2);
    }
    static void unregister_page(void*) { ++g_unreg; }
    static void clear_error() { ++g_clear; }
};
}  // namespace

extern "C" void host_page_run(int fail, int* out) {
    g_fail = fail;
    g_reg = g_unreg = g_clear = 0;
    eup::HostPage<Api> p;
    out[0] = p.open();
    if (out[0]) p.host[511] = 1.0;
    out[1] = p.open();
    p.close();
    p.close();
    out[2] = g_reg;
    out[3] = g_unreg;
    out[4] = g_clear;
    out[5] = p.host != nullptr;
    out[6] = p.dev != nullptr;
}
