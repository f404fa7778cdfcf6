// What kernels are given of a caller's memory: only pages that are there and that
// they may use.  The pages of an untouched output are there before the kernel is
// launched; an output that may not be written goes through device memory.
#include "fake_cudart.h"

#include "texpresso_gb300.h"

#include <sys/mman.h>
#include <unistd.h>

constexpr uint32_t W = 1024, H = 512;
constexpr size_t kImage = 4 * (size_t)W * H;

uint8_t *map(size_t n, int prot) {
    void *p = mmap(nullptr, n, prot, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    CHECK(p != MAP_FAILED);
    return static_cast<uint8_t *>(p);
}

size_t resident(uint8_t *p, size_t n) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    std::vector<unsigned char> v((n + page - 1) / page);
    CHECK(mincore(p, n, v.data()) == 0);
    size_t k = 0;
    for (unsigned char c : v) k += c & 1;
    CHECK(k <= v.size());
    return v.size() - k;  // pages that are missing
}

int main() {
    const size_t size = tx_compressed_size(TX_FORMAT_BC3, W, H);
    tx_params p;
    tx_params_default(&p);
    p.algorithm = TX_RANGE_FIT;
    const uint8_t *given_in = nullptr;
    uint8_t *given_out = nullptr, *output = nullptr;
    size_t missing = 0, out_bytes = 0;
    bool stop = false;  // let no copy out follow the kernel
    fake::kernel_body = [&](const std::string &name, dim3, void **args) -> std::function<void()> {
        const bool decode = name.find("k_decode") != std::string::npos;
        if (decode || name.find("k_range") != std::string::npos) {
            given_in = *static_cast<const uint8_t **>(args[0]);  // (SrcDesc::base comes first)
            given_out = *static_cast<uint8_t **>(args[decode ? 6 : 2]);
            missing = resident(output, out_bytes);
            if (stop) fake::fail_after["cudaMemcpyAsync"] = 0;
        }
        return nullptr;
    };
    for (int decode = 0; decode < 2; ++decode) {
        auto run = [&](uint8_t *in, uint8_t *out) {
            output = out;
            out_bytes = decode ? kImage : size;
            given_in = given_out = nullptr;
            const int rc = decode ? tx_decompress(TX_FORMAT_BC3, in, size, W, H, out, kImage)
                                  : tx_compress(TX_FORMAT_BC3, in, kImage, W, H, &p, out, size);
            fake::fail_after.clear();
            CHECK(given_out != nullptr);
            CHECK(fake::in_flight() == 0);
            return rc;
        };
        uint8_t *in = map(kImage, PROT_READ | PROT_WRITE), *out = map(kImage, PROT_READ | PROT_WRITE);
        CHECK(run(in, out) == TX_OK);
        CHECK(given_in == in && given_out == out);
        CHECK(missing == 0);
        uint8_t *fixed = map(kImage, PROT_READ);
        stop = true;
        CHECK(run(in, fixed) == TX_ERR_CUDA);
        CHECK(given_out != fixed);
        stop = false;
        CHECK(run(fixed, out) == TX_OK);  // an input may be read-only
        CHECK(given_in == fixed && given_out == out);
    }
    return 0;
}
