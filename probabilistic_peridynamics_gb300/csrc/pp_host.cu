// pp_host.cu -- host memory: page-locking of caller arrays for copies to and
// from the device, and threaded copies of large arrays.
//
// The library links its own (static) CUDA runtime, so a failed registration
// leaves its error in this runtime, where it is cleared here, and not in the
// runtime of the caller (torch's, for the Python integrators), whose next
// launch check would otherwise report it at an unrelated call.  The pages
// are registered with the device's primary context, which every runtime in
// the process shares, so copies issued by the caller's runtime see them as
// page-locked.
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

#include "pp_common.cuh"

namespace {

// work(a, b) over [0, n) on up to eight threads, in pieces of at least
// `least`.  Writing a fresh 205 MB array is bound by its page faults: 19 ms on
// one thread of the host.
template <class Work>
void in_parallel(int64_t n, int64_t least, Work&& work) {
    int64_t parts = n / (least > 0 ? least : 1);
    const int64_t most = std::thread::hardware_concurrency();
    if (parts > most) parts = most;
    if (parts > 8) parts = 8;
    if (parts < 2) {
        work(0, n);
        return;
    }
    const int64_t size = (n + parts - 1) / parts;
    std::vector<std::thread> threads;
    int64_t done = size;  // the caller's own piece
    try {
        threads.reserve(parts);
        for (; done < n; done += size) {
            const int64_t a = done, b = done + size < n ? done + size : n;
            threads.emplace_back([&work, a, b] { work(a, b); });
        }
    } catch (const std::exception&) {
        // no more threads: the rest is the caller's
        work(done, n);
    }
    work(0, size < n ? size : n);
    for (std::thread& t : threads) t.join();
}

}  // namespace

extern "C" int pp_host_register(void* ptr, size_t bytes) {
    if (!ptr || bytes == 0) return PP_ERROR_INVALID_VALUE;
    if (cudaHostRegister(ptr, bytes, cudaHostRegisterDefault) != cudaSuccess) {
        (void)cudaGetLastError();  // non-sticky: clear it
        return PP_ERROR_CUDA;
    }
    return PP_SUCCESS;
}

extern "C" int pp_host_unregister(void* ptr) {
    if (!ptr) return PP_ERROR_INVALID_VALUE;
    if (cudaHostUnregister(ptr) != cudaSuccess) {
        (void)cudaGetLastError();
        return PP_ERROR_CUDA;
    }
    return PP_SUCCESS;
}

extern "C" int pp_host_copy(void* dst, const void* src, size_t bytes) {
    if (bytes == 0) return PP_SUCCESS;
    if (!dst || !src) return PP_ERROR_INVALID_VALUE;
    in_parallel((int64_t)bytes, 4 << 20, [&](int64_t a, int64_t b) {
        std::memcpy(static_cast<char*>(dst) + a, static_cast<const char*>(src) + a, (size_t)(b - a));
    });
    return PP_SUCCESS;
}

extern "C" int pp_host_local_rows(const int32_t* src, int64_t rows, int64_t width, int64_t columns,
                                  int64_t offset, int64_t* dst) {
    if (rows < 0 || columns < 0 || columns > width) return PP_ERROR_INVALID_VALUE;
    if (rows == 0 || columns == 0) return PP_SUCCESS;
    if (!src || !dst) return PP_ERROR_INVALID_VALUE;
    in_parallel(rows, (1 << 18) / columns + 1, [&](int64_t a, int64_t b) {
        for (int64_t r = a; r < b; ++r) {
            const int32_t* s = src + r * width;
            int64_t* d = dst + r * columns;
            for (int64_t c = 0; c < columns; ++c) d[c] = s[c] >= 0 ? s[c] - offset : -1;
        }
    });
    return PP_SUCCESS;
}
