// The allocation-free batch launch does all set-up in its first call on a device:
// whatever that call compresses, later calls load no kernel and set no attribute.
#include "fake_cudart.h"

#include "texpresso_gb300.h"

#include <algorithm>

int main() {
    static uint8_t src[64 * 64 * 4], dst[64 * 64];
    auto item = [](int format, int algorithm) {
        tx_batch_item it{};
        it.src = src;
        it.src_pitch = 64 * 4;
        it.width = it.height = 64;
        it.format = format;
        it.channels = 4;
        tx_params_default(&it.params);
        it.params.algorithm = algorithm;
        it.dst = dst;
        return it;
    };
    const tx_batch_item first = item(TX_FORMAT_BC3, TX_CLUSTER_FIT);
    CHECK(tx_batch_launch_noalloc(&first, 1, nullptr) == TX_OK);
    const std::vector<std::string> ready = [] {
        std::vector<std::string> v = fake::prepared;
        v.insert(v.end(), fake::launched.begin(), fake::launched.end());
        return v;
    }();
    const std::map<std::string, int> before = fake::calls;
    const size_t n = fake::launched.size();
    std::vector<tx_batch_item> all;
    for (int f = TX_FORMAT_BC1; f <= TX_FORMAT_BC5; ++f)
        for (int a = TX_RANGE_FIT; a <= TX_ITERATIVE_CLUSTER_FIT; ++a) all.push_back(item(f, a));
    CHECK(tx_batch_launch_noalloc(all.data(), all.size(), nullptr) == TX_OK);
    CHECK(fake::launched.size() > n + 6);
    for (size_t k = n; k < fake::launched.size(); ++k) {
        if (std::find(ready.begin(), ready.end(), fake::launched[k]) == ready.end()) {
            fprintf(stderr, "not set up by the first call: %s\n", fake::launched[k].c_str());
            return 1;
        }
    }
    for (const char *name : {"cudaFuncSetAttribute", "cudaMalloc", "cudaMallocFromPoolAsync"}) {
        if (fake::calls[name] != (before.count(name) ? before.at(name) : 0)) {
            fprintf(stderr, "called again: %s\n", name);
            return 1;
        }
    }
    return 0;
}
