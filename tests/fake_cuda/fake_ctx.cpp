#include "fake_ctx.h"

#include "fake_cuda.h"
#include "internal.h"

namespace fake {
std::atomic<int> live{0}, recycled{0}, recycled_busy{0}, destroyed_elsewhere{0}, fail_after{-1};
std::thread::id main_thread = std::this_thread::get_id();
}  // namespace fake

static void queue_work(gnss_ctx *c, void *stream) {
    c->queued++;
    fake::enqueue(static_cast<cudaStream_t>(stream), [c] { c->queued--; });
}

// C linkage comes from the declarations in gnss_b200.h
gnss_status gnss_create(const gnss_config *cfg, gnss_ctx **out) {
    if (cfg->nx < 8) return GNSS_ERR_INVALID;
    if (cudaSetDevice(cfg->device) != cudaSuccess) return GNSS_ERR_CUDA;
    *out = new gnss_ctx;
    (*out)->cfg = *cfg;
    fake::live++;
    return GNSS_OK;
}
gnss_status gnss_destroy(gnss_ctx *c) {
    cudaSetDevice(c->cfg.device);
    fake::drain_all();   // cudaFree waits for the device
    if (std::this_thread::get_id() != fake::main_thread) fake::destroyed_elsewhere++;
    fake::live--;
    delete c;
    return GNSS_OK;
}
bool gnss_recycle(gnss_ctx *c, const gnss_config *cfg) {
    if (c->cfg.nx != cfg->nx) return false;
    fake::recycled++;
    if (c->queued) fake::recycled_busy++;
    c->cfg = *cfg;
    return true;
}
gnss_status gnss_reset_run(gnss_ctx *c, void *stream) { queue_work(c, stream); return GNSS_OK; }
gnss_status gnss_step(gnss_ctx *c, const gnss_fields *, const gnss_fields *, int, void *stream) {
    if (fake::fail_after >= 0 && fake::fail_after-- == 0) return GNSS_ERR_CUDA;
    queue_work(c, stream);
    return GNSS_OK;
}
gnss_status gnss_dealias(gnss_ctx *c, void *, void *stream) { queue_work(c, stream); return GNSS_OK; }
gnss_status gnss_stats(gnss_ctx *, const gnss_fields *, double *out, void *stream) {
    for (int i = 0; i < GNSS_NSTATS; ++i) out[i] = i;
    return cudaStreamSynchronize(static_cast<cudaStream_t>(stream)) == cudaSuccess ? GNSS_OK : GNSS_ERR_CUDA;
}
gnss_status gnss_attach_scratch(gnss_ctx *, void *, size_t) { return GNSS_OK; }
size_t gnss_scratch_bytes(const gnss_ctx *) { return 4096; }
size_t gnss_workspace_bytes(const gnss_ctx *) { return 4096; }
gnss_status gnss_set_option(gnss_ctx *, int, int) { return GNSS_OK; }
long long gnss_launch_count(const gnss_ctx *) { return 0; }
size_t gnss_batch_scratch_bytes(const gnss_ctx *) { return 4096; }
bool gnss_batch_supported(const gnss_ctx *) { return false; }
gnss_status gnss_step_batch(gnss_ctx *const *, int, const gnss_fields *, const gnss_fields *, size_t, void *, size_t, int,
                            void *) {
    return GNSS_ERR_UNSUPPORTED;
}
