// A page of host memory that the device writes to.  Api: the four CUDA calls (true: done), so that
// tests can let them fail.
#pragma once
#include <stddef.h>

#include <cstdlib>

namespace eup {

constexpr size_t kHostPage = 4096;

template <typename Api>
struct HostPage {
    double* host = nullptr;
    double* dev = nullptr;  // where the device writes it; null: there is no page

    // A page of our own, registered: 0.3 ms, and 0.19 to release, where the first cudaMallocHost of
    // a process takes 1.5 and the last cudaFreeHost 0.5.  false: nothing is held and no error
    // is left behind.
    bool open() {
        if (dev) return true;
        host = static_cast<double*>(std::aligned_alloc(kHostPage, kHostPage));
        if (!host) return false;
        void* d = nullptr;
        const bool registered = Api::register_page(host, kHostPage);
        if (registered && Api::device_pointer(host, &d) && d) {
            dev = static_cast<double*>(d);
            return true;
        }
        if (registered) Api::unregister_page(host);
        Api::clear_error();
        std::free(host);
        host = nullptr;
        return false;
    }
    void close() {
        if (dev) Api::unregister_page(host);
        std::free(host);
        host = dev = nullptr;
    }
};

}  // namespace eup
