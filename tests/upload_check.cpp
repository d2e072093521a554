// Uploads from pageable memory (visualmesh_b200/csrc/upload.hpp) and the libm tables without a GPU: the copy to the device is a memcpy
// here, and pthread_create fails from the n-th call on when asked to.
//
//   upload_check copies [first thread that cannot be started]     every byte arrives, from several calling threads at once
//   upload_check tables [first thread that cannot be started]     the table's words are those of the host's libm
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <cstdio>
#include <cstdlib>
#include <string>

#include "../visualmesh_b200/csrc/upload.hpp"
#include "../visualmesh_b200/csrc/libm_tables.hpp"

static std::atomic<int> g_created{0};
static int g_first_refused = 1 << 30;

extern "C" int pthread_create(pthread_t* thread, const pthread_attr_t* attr, void* (*start)(void*), void* arg) {
    using Real        = int (*)(pthread_t*, const pthread_attr_t*, void* (*) (void*), void*);
    static Real real  = reinterpret_cast<Real>(dlsym(RTLD_NEXT, "pthread_create"));
    if (g_created.fetch_add(1) >= g_first_refused) return EAGAIN;
    return real(thread, attr, start, arg);
}

extern "C" cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(dst, src, n);
    return cudaSuccess;
}

static bool upload_once(unsigned seed) {
    // around the 16-byte stores, the 64-byte steps and the slices; pageable frames lie 256 bytes apart in the staging buffer
    static const size_t sizes[] = {1, 15, 16, 17, 63, 64, 65, 1000, vm::UPLOAD_SLICE - 1, vm::UPLOAD_SLICE, vm::UPLOAD_SLICE + 1, 3 * vm::UPLOAD_SLICE + 77};
    std::vector<std::vector<uint8_t>> frames;
    std::vector<size_t> at;
    size_t total = 0;
    for (unsigned f = 0; f < 5; ++f) {
        const size_t n = sizes[(seed * 5 + f * 7) % (sizeof(sizes) / sizeof(sizes[0]))], shift = (seed + f) % 17;
        frames.emplace_back(n + shift);
        for (size_t i = 0; i < frames.back().size(); ++i) frames.back()[i] = static_cast<uint8_t>(seed * 31 + f * 7 + i * 13 + (i >> 8));
        at.push_back(total);
        total += (n + 255) / 256 * 256;
    }
    std::vector<uint8_t> staging(total + 16, 0xEE), device(total, 0xDD);
    std::shared_ptr<vm::UploadHelpers> helpers = vm::UploadHelpers::get();
    vm::Upload upload(helpers.get(), device.data(), nullptr);
    for (unsigned f = 0; f < frames.size(); ++f) {
        const size_t shift = (seed + f) % 17;
        upload.job.add(frames[f].data() + shift, at[f], frames[f].size() - shift);
    }
    upload.start(staging.data() + seed % 16);
    upload.pump();
    upload.finish();
    for (unsigned f = 0; f < frames.size(); ++f) {
        const size_t shift = (seed + f) % 17;
        if (std::memcmp(device.data() + at[f], frames[f].data() + shift, frames[f].size() - shift) != 0) return false;
    }
    return true;
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (argc > 2) g_first_refused = std::atoi(argv[2]);
    if (what == "copies") {
        // the helpers start with the first upload and, kept here, serve all that follow
        std::shared_ptr<vm::UploadHelpers> kept = vm::UploadHelpers::get();
        g_first_refused                         = 1 << 30;
        std::atomic<int> wrong{0};
        std::vector<std::thread> callers;
        for (unsigned t = 0; t < 3; ++t)
            callers.emplace_back([&wrong, t] {
                for (unsigned i = 0; i < 40; ++i)
                    if (!upload_once(100 * t + i)) ++wrong;
            });
        for (auto& c : callers) c.join();
        std::printf("%d wrong\n", wrong.load());
        return wrong.load() == 0 ? 0 : 1;
    }
    if (what == "tables") {
        const std::vector<uint32_t> packed = vm::libm::build(vm::libm::SIN);
        long wrong = 0;
        for (size_t w = 0; w < packed.size(); w += 997) {
            const uint32_t bits = vm::libm::FIRST_BITS[vm::libm::SIN] + static_cast<uint32_t>(w) * 16u + w % 16;
            float x;
            std::memcpy(&x, &bits, sizeof(x));
            const float y = vm::libm::evaluate(vm::libm::SIN, x);
            uint32_t yb;
            std::memcpy(&yb, &y, sizeof(yb));
            wrong += (packed[w] >> (2 * (w % 16)) & 3u) != (yb & 3u);
        }
        std::printf("%ld wrong\n", wrong);
        return wrong == 0 ? 0 : 1;
    }
    return 2;
}
