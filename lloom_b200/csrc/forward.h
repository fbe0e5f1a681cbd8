// C++ interface behind the C ABI's forward entries: what the ABI unit offers to the package's own host layers (the
// Python binding), which know more about a call than the C entries can say -- the element types of activations and
// outputs, and that the weights were in place before the stream's previous kernel started (launch overlap).
#pragma once

#include <stdint.h>

#include "../../include/lloom_b200.h"

namespace lloom {

// The setting of lloom_b200_set_launch_overlap: 1 on, 0 off, -1 neither (the host layer decides call by call).
int launch_overlap();

struct FwdIo {
    int x_type = LLOOM_F32, y_type = LLOOM_F32;  // LLOOM_F32 / LLOOM_F16 / LLOOM_BF16
    // The call's kernels may start before their stream predecessor has finished; they read nothing but weights until it
    // has.  Only for weights that no work still in flight writes.
    bool overlap = false;
};

// All return a status code; shapes, pointers and workspace are checked as by the C entries of the same name.
// lloom_b200_qmatmul_fwd (w_image == nullptr, store == LLOOM_STORE_PLAIN), _image and _store in one.
int qmatmul_forward(int w_dtype, const void *w_blocks, const void *w_image, const void *x, void *y, int64_t m, int64_t n, int64_t k,
                    int64_t ldy, int store, void *workspace, int64_t workspace_bytes, void *stream, const FwdIo &io);
int qmatmul_forward_group(int w_dtype, int n_mats, const void *const *w_blocks, const void *x, float *const *ys, const int64_t *ns,
                          const int64_t *ldys, const int *stores, int64_t m, int64_t k, void *workspace, int64_t workspace_bytes,
                          void *stream, const FwdIo &io);
// ids: 32-bit, or 64-bit of which the low half counts
int indexed_moe_forward(int w_dtype, const void *w_experts, int64_t n_experts, int64_t n, int64_t k, const float *x, int64_t batch,
                        int64_t in_dim1, const void *ids, bool ids64, int64_t topk, float *out, void *workspace,
                        int64_t workspace_bytes, void *stream, const FwdIo &io);
int get_rows(int dtype, const void *blocks, int64_t rows, int64_t hidden, const void *ids, bool ids64, int64_t n_ids, float *out,
             void *stream, bool overlap);

}  // namespace lloom
