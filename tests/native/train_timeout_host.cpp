// The training loop's host code when a tensor-core kernel reports a timeout or
// a launch fails: the library's own code on the host stand-in of the CUDA
// runtime, with launches that only count. Prints one line per step; test-only.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../../grrt_b200/csrc/device/mlp_fused.h"
#include "../../grrt_b200/csrc/device/surrogate.h"
#include "../../grrt_b200/csrc/device/umma_gemm.h"
#include "../../include/grrt_surrogate.h"
#include "fake_cuda.h"

namespace {
int steps_run = 0;        // training steps that the GPU finished
int timeout_step = -1;    // the step whose GEMMs time out (and those after it)
int enqueue_fail = -1;    // the weight-gradient launch that fails
int weight_gemms = 0;
std::map<cudaStream_t, unsigned long long> last_work;  // queue position behind a stream's last launch

cudaError_t work(cudaStream_t s, fake::Op op = [] {}) {
    fake::enqueue(std::move(op));
    if (!fake::capture) last_work[s] = fake::queued;
    return cudaSuccess;
}
}  // namespace

namespace grrt_b200 {
using bf = __nv_bfloat16;

cudaError_t umma_gemm_bf16(const bf*, int, const bf*, int, int, int, int, int, const GemmEpilogue&, int* err,
                           cudaStream_t s) {
    return work(s, [=] {
        if (timeout_step >= 0 && steps_run >= timeout_step) *err = 3;
    });
}
cudaError_t umma_gemm_tn_bf16(const bf*, int, const bf*, int, int, int, int, int, const GemmEpilogue&, int*,
                              cudaStream_t s) {
    return ++weight_gemms == enqueue_fail ? cudaErrorLaunchFailure : work(s);
}

namespace surr {
bool make_mlp_maps(bf* const*, const bf*, MlpMaps*) { return true; }
cudaError_t launch_trace_dataset(const DevScene*, int, int, int, float*, float*, unsigned*, DevStats*, cudaStream_t s) {
    return work(s);
}
cudaError_t launch_gather(const float*, const float*, size_t, int, const unsigned*, float*, float*, cudaStream_t s) {
    return work(s);
}
cudaError_t launch_layer1_fwd(const float*, int, const float*, float*, bf*, cudaStream_t s) { return work(s); }
cudaError_t launch_loss(const float*, const float*, int, LossWeights, bf*, float* loss, cudaStream_t s) {
    return work(s, [=] { *loss = 1.0f + static_cast<float>(steps_run); });
}
cudaError_t launch_colsum(const bf*, int, int, int, float*, int, float*, cudaStream_t s) { return work(s); }
cudaError_t launch_layer1_bwd(const bf*, const float*, int, float*, int, float*, cudaStream_t s) { return work(s); }
cudaError_t launch_reduce_splits(const float*, int, size_t, float*, cudaStream_t s) { return work(s); }
cudaError_t launch_adam(float*, const float*, float*, float*, size_t, const unsigned*, const float*, float, float,
                        float, cudaStream_t s) {
    return work(s);
}
cudaError_t launch_finish_step(const float* loss, unsigned* step, float* hist, int cap, cudaStream_t s) {
    return work(s, [=] {
        if (static_cast<int>(*step) < cap) hist[*step] = *loss;
        ++*step;
        ++steps_run;
    });
}
cudaError_t launch_set_float(float* p, float v, cudaStream_t s) {
    return work(s, [=] { *p = v; });
}
cudaError_t launch_cast_weights(const float*, bf* const*, bf* const*, bf*, bf*, cudaStream_t s) { return work(s); }
}  // namespace surr
}  // namespace grrt_b200

namespace {

void train(GRRTSurrogate* s, int steps, const char* step) {
    std::vector<float> loss(static_cast<size_t>(steps), -7.0f);
    const int before = steps_run;
    const int rc = grrt_surrogate_train(s, steps, 128, 1e-3, loss.data());
    int filled = 0;
    bool drained = true;
    for (float v : loss) filled += v != -7.0f;
    for (const auto& [stream, n] : last_work) drained = drained && fake::waited[stream] >= n;
    const char* e = grrt_surrogate_error(s);
    std::printf("%s rc=%d steps=%d filled=%d last=%g drained=%d error=%s\n", step, rc, steps_run - before, filled,
                loss.back(), drained, e ? e : "none");
}

}  // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const int steps = argc > 2 ? std::atoi(argv[2]) : 80;
    GRRTSurrogate* s = grrt_surrogate_create(1);
    GRRTParams cam;
    std::memset(&cam, 0, sizeof(cam));
    cam.disk_enabled = 1;
    if (!s || grrt_surrogate_generate(s, &cam, 1, 16) != 0) return 3;
    if (what == "timeout") {
        timeout_step = 2;
        train(s, steps, "bad");
        timeout_step = -1;
        train(s, steps, "after");
    } else if (what == "launch") {
        enqueue_fail = 6;  // in the second step's capture or after the first one's
        train(s, steps, "bad");
        enqueue_fail = -1;
        train(s, steps, "after");
    } else if (what == "eager") {
        enqueue_fail = 3;
        train(s, steps, "bad");
        train(s, steps, "after");
    } else {
        return 2;
    }
    grrt_surrogate_destroy(s);
    return 0;
}
