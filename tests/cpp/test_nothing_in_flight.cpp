// Host-buffer calls that fail part of the way: when they return, no copy or kernel
// that uses the caller's buffers is still in flight, whichever call failed.
#include "fake_cudart.h"

#include "texpresso_gb300.h"

int main() {
    constexpr uint32_t W = 64, H = 512;  // 128 rows of blocks: bands on three streams
    std::vector<uint8_t> image(4 * W * H + 8), blocks(W * H + 16);
    uint8_t *odd = blocks.data() + 1;  // not 8-byte aligned
    const size_t size = tx_compressed_size(TX_FORMAT_BC3, W, H);
    auto compress = [&] {
        return tx_compress(TX_FORMAT_BC3, image.data(), 4 * W * H, W, H, nullptr, blocks.data(), size);
    };
    auto decompress = [&] { return tx_decompress(TX_FORMAT_BC3, odd, size, W, H, image.data(), 4 * W * H); };
    auto block = [&] { return tx_compress_block_masked(TX_FORMAT_BC3, image.data(), 0xFFFFu, nullptr, blocks.data(), 16); };
    auto decompress_block = [&] { return tx_decompress_block(TX_FORMAT_BC3, blocks.data(), 16, image.data()); };
    const std::pair<const char *, std::function<int()>> entry[] = {
        {"tx_decompress", decompress}, {"tx_compress", compress}, {"tx_compress_block_masked", block},
        {"tx_decompress_block", decompress_block}};
    int device = 0;
    for (int tables = 0; tables < 2; ++tables) {
        for (const auto &e : entry) {
            for (const char *api : {"cudaMalloc", "cudaMemcpyAsync", "launch", "cudaEventRecord", "cudaStreamWaitEvent"}) {
                cudaSetDevice(device++);  // a device that holds no buffers yet
                fake::host_page_tables = tables;
                CHECK(tx_compress_block_masked(TX_FORMAT_BC3, image.data(), 0, nullptr, blocks.data(), 16) == TX_OK);
                for (int n = 0;; ++n) {
                    fake::fail_after[api] = n;
                    const int rc = e.second();
                    fake::fail_after.clear();
                    if (fake::in_flight()) {
                        fprintf(stderr, "%s, %s number %d fails (host page tables: %d): %zu operations in flight\n", e.first,
                                api, n + 1, tables, fake::in_flight());
                        return 1;
                    }
                    if (rc == TX_OK) break;  // it makes no more than n of these calls
                    CHECK(n < 64);
                }
            }
        }
    }
    return 0;
}
