// Which kernel an FP64 thin-disk batch renders with, and what happens to its
// schedule when the autotuner or an allocation fails: the library's own batch
// code on the host stand-in of the CUDA runtime, with launches that only note
// their name. Prints one line per step; test-only.
#include <cstdio>
#include <cstring>
#include <string>

#include "../../grrt_b200/csrc/device/render_launch.h"
#include "../../include/grrt_b200.h"
#include "fake_cuda.h"

namespace {
std::string ran;        // the last batch kernel that ran
int launches = 0;       // batch launches enqueued or captured so far
int fail_at = 0;        // the launch that fails (0: none)
double pixel_ms = 2.0, sample_ms = 1.0, mixed_ms = 0.5;

cudaError_t note(const char* name, double ms) {
    if (++launches == fail_at) return cudaErrorLaunchFailure;
    fake::enqueue([=] {
        ran = name;
        fake::now_ms += ms;
    });
    return cudaSuccess;
}
}  // namespace

namespace grrt_b200 {
size_t mixed_scratch_bytes_for(size_t n) { return 1024 + 60 * n; }
cudaError_t launch_thin_batch(const DevBatch&, float4*, unsigned*, DevStats*, int, int, cudaStream_t) {
    return note("pixels", pixel_ms);
}
cudaError_t launch_thin_fp64_batch(const DevBatch&, float4*, unsigned*, DevStats*, void*, size_t, int, cudaStream_t) {
    return note("samples", sample_ms);
}
cudaError_t launch_thin_mixed_batch(const DevBatch&, bool, float4*, unsigned*, DevStats*, void*, size_t, int,
                                    cudaStream_t) {
    return note("mixed", mixed_ms);
}
int thin_batch_max_blocks_per_sm(int block) { return 512 / block; }
int fp64_batch_max_blocks_per_sm() { return 4; }
int mixed_batch_max_blocks_per_sm() { return 5; }
}  // namespace grrt_b200

namespace {

GRRTBatch* make(int cameras, int w, int h) {
    GRRTParams p[8];
    std::memset(p, 0, sizeof(p));
    for (int i = 0; i < cameras; ++i) {
        p[i].width = w;
        p[i].height = h;
        p[i].disk_enabled = 1;
        p[i].samples_per_pixel = 1;
    }
    return grrt_batch_create(p, cameras);
}

void render(GRRTBatch* b, const char* step) {
    const size_t before = fake::used;
    ran = "nothing";
    const int rc = grrt_batch_render(b, std::vector<float*>(8, nullptr).data());
    int chunk, order, bps, block;
    double tol, rf;
    grrt_batch_get_schedule(b, &chunk, &order, &bps);
    grrt_batch_get_tuning(b, &block, &tol, &rf);
    std::printf("%s rc=%d ran=%s schedule=%d,%d,%d block=%d took=%s\n", step, rc, ran.c_str(), chunk, order, bps, block,
                fake::used > before ? "memory" : "none");
}

}  // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const char* cache = argc > 2 ? argv[2] : nullptr;
    GRRTBatch* b = make(2, 40, 30);
    if (what == "default") {
        render(b, "first");
    } else if (what == "schedule") {
        grrt_batch_set_schedule(b, 256, GRRT_BATCH_ORDER_ROUND_ROBIN, 0);
        render(b, "set");
    } else if (what == "tolerance") {
        grrt_batch_set_tuning(b, 128, 1e-6, 4.0);
        render(b, "set");
    } else if (what == "block") {
        grrt_batch_set_tuning(b, 64, 3e-6, 3.0);
        render(b, "set");
        grrt_batch_set_tuning(b, 128, 3e-6, 3.0);
        render(b, "back");
    } else if (what == "mixed_autotune" || what == "mixed_cached") {
        grrt_batch_set_precision(b, GRRT_FORM_MIXED);
        double ms = 0;
        std::printf("autotune rc=%d\n", grrt_batch_autotune(b, cache, &ms));
        render(b, "mixed");
        grrt_batch_set_precision(b, GRRT_FORM_FP64);
        render(b, "fp64");
    } else if (what == "fp64_autotune" || what == "fp64_cached") {
        pixel_ms = 0.5;  // the tuner finds the pixels faster
        double ms = 0;
        std::printf("autotune rc=%d\n", grrt_batch_autotune(b, cache, &ms));
        render(b, "fp64");
        grrt_batch_set_precision(b, GRRT_FORM_MIXED);
        grrt_batch_autotune(b, nullptr, &ms);
        grrt_batch_set_precision(b, GRRT_FORM_FP64);
        render(b, "again");
    } else if (what == "failed_autotune" || what == "failed_mixed_autotune") {
        if (what == "failed_mixed_autotune") grrt_batch_set_precision(b, GRRT_FORM_MIXED);
        fail_at = 3;
        double ms = 0;
        std::printf("autotune rc=%d\n", grrt_batch_autotune(b, cache, &ms));
        fail_at = 0;
        grrt_batch_set_precision(b, GRRT_FORM_FP64);
        render(b, "after");
    } else if (what == "no_room") {
        // two cameras of 2048 x 2048: 0.5 GB of sample scratch
        grrt_batch_destroy(b);
        b = make(2, 2048, 2048);
        fake::room = size_t(300) << 20;
        render(b, "full");
        fake::room = size_t(180) << 30;
        render(b, "freed");
        render(b, "replay");
    } else if (what == "little_room") {
        grrt_batch_destroy(b);
        b = make(2, 2048, 2048);
        fake::room = size_t(1) << 30;
        render(b, "little");
        grrt_batch_set_schedule(b, 256, GRRT_BATCH_ORDER_SAMPLES, 0);
        render(b, "asked");
    } else if (what == "too_many") {
        // 1.05 GB of sample scratch
        grrt_batch_destroy(b);
        b = make(5, 2048, 1760);
        render(b, "large");
    } else {
        return 2;
    }
    grrt_batch_destroy(b);
    return 0;
}
