// FP64 instantiation of the fused path (kernels in pfag_fused_impl.cuh).
#include "pfag_fused_impl.cuh"

int pfag_fused_alloc_f64(pfag_ctx *c) { return fused_alloc_t<double>(c); }
int pfag_fused_upload_f64(pfag_ctx *c) { return fused_upload_t<double>(c); }
int pfag_fused_step_f64(pfag_ctx *c) { return fused_step_t<double>(c); }
int pfag_fused_recentre_f64(pfag_ctx *c) { return fused_recentre_t<double>(c); }
int pfag_fused_capture_f64(pfag_ctx *c, bool beside, cudaGraph_t *g, long *launches) {
    return fused_capture_t<double>(c, beside, g, launches);
}
int pfag_fused_step_part_f64(pfag_ctx *c, int part) { return fused_step_part_t<double>(c, part); }
