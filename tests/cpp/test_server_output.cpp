// A served job's output is written on completion: the compression steps write to
// device memory, and the output gets all its blocks at once after the last of them.
#include "fake_cudart.h"

#include "texpresso_gb300.h"

int main() {
    constexpr uint32_t W = 512, H = 384;
    std::vector<uint8_t> image(4 * W * H), room(W * H * 2 + 64);
    bool in_steps = false;
    int stores = 0, steps = 0, steps_at_store = 0;
    uint8_t *output = nullptr;
    size_t size = 0;
    fake::kernel_body = [&](const std::string &name, dim3, void **args) -> std::function<void()> {
        if (name.find("k_store") != std::string::npos) {
            return [&] { ++stores; steps_at_store = steps; };
        }
        if (name.find("k_batch_") == std::string::npos) return nullptr;
        // the items are copied to the device before the kernel runs
        const uint8_t *items = *static_cast<const uint8_t **>(args[0]);  // (BatchQueue::items comes first)
        return [&, items] {
            ++steps;
            for (size_t k = 0; k < 4096; ++k) {
                uint8_t *p;
                memcpy(&p, items + 8 * k, 8);
                in_steps = in_steps || (p >= output && p < output + size);
            }
        };
    };
    tx_server_config cfg;
    tx_server_default_config(&cfg);
    cfg.step_blocks = 4096;  // several steps for each job
    cfg.min_share = 1024;
    tx_server *server = nullptr;
    CHECK(tx_server_create(&cfg, &server) == TX_OK);
    for (int format = TX_FORMAT_BC1; format <= TX_FORMAT_BC5; ++format) {
        for (int offset : {0, 1}) {
            tx_server_request r{};
            r.rgba = image.data();
            r.width = W;
            r.height = H;
            r.format = format;
            tx_params_default(&r.params);
            r.mips = 1;
            {
                std::lock_guard<std::recursive_mutex> lk(fake::mu);
                stores = steps = 0;
                r.output = output = room.data() + (16 - (uintptr_t)room.data() % 16) + offset;
                r.output_len = size = tx_chain_compressed_size(format, W, H, 1);
            }
            uint64_t id;
            CHECK(tx_server_submit(server, &r, &id) == TX_OK);
            CHECK(tx_server_wait(server, id, 20000, nullptr) == TX_OK);
            std::lock_guard<std::recursive_mutex> lk(fake::mu);
            CHECK(!in_steps);
            CHECK(steps >= 3 && stores == 1 && steps_at_store == steps);
        }
    }
    tx_server_destroy(server);
    return 0;
}
