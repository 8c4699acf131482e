// skml_train_step: the launch sequence of one training step behind a single C call.
// Reference: ml/algorithm/GeneralizedLinearModel.scala:116-123 (trainOneIteration =
// computeGradient + aggregateAndUpdate); here the whole iteration is four kernel launches
// (coefficients, column sums, fused compress, fused decode + update) issued back to
// back on one stream with no host round trip.
#include <cuda_runtime.h>

#include "skml_api.h"

// The batch arrays (rowptr, cols, vals, labels) are read by the gradient kernels only (a local-id
// batch's column list also by the compress kernel); a feeder that recycles them waits for this event.
static int batch_consumed(const SkmlStepArgs* a, cudaStream_t stream) {
    if (!a->grad_done_event) return 0;
    return (int)cudaEventRecord((cudaEvent_t)a->grad_done_event, stream);
}

// The gradient's way into the model: through the fused compress and decode kernels, or through a baseline's codes.
// `n_bound`: as many non-zeros there are (0: not known here, n_max at most). `batch_keys`: keys and count lie in the batch's own buffers, which are the feeder's again once they are read.
static int apply_gradient(SkmlStepArgs* a, const int* keys, const long long* meta, float* vals, float* dense_vals, long long n_bound,
                          bool batch_keys, void* stream) {
    if (a->coded) {
        const SkmlCodedArgs& c = *a->coded;
        int rc = 0;
        if (c.kind == 1) {
            rc = skml_fixedpoint_pack(vals, meta, a->n_max, (int)c.bits, c.seed, (double*)c.scratch, c.codes, c.norm, stream);
            if (!rc) rc = skml_fixedpoint_unpack_scatter(nullptr, keys, c.codes, c.norm, meta, a->n_max, c.code_stride, 1, (int)c.bits, vals, stream);
        } else if (c.kind == 2) {
            rc = skml_zipml_pack(vals, meta, n_bound > 0 && n_bound < a->n_max ? n_bound : a->n_max, (int)c.bits, c.scratch, c.scratch_bytes, c.splits, c.mids, c.zip_meta, c.range, c.codes,
                                 a->status, stream);
            if (!rc) rc = skml_zipml_unpack_scatter(nullptr, keys, c.codes, c.mids, meta, a->n_max, c.code_stride, 1, (int)c.bits, vals,
                                                    a->status, stream);
        }
        if (rc) return rc;
        rc = skml_update_sparse(a->w, c.adam_m, c.adam_v, keys, vals, meta, a->n_max, 1.f, c.adam_v != nullptr, (float)a->lr,
                                (float)a->adam_scale, (int)c.adam_stride, a->status, stream);
        if (rc) return rc;
        return (int)cudaMemcpyAsync(a->loss_out, a->partials, 4 * sizeof(double), cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
    }
    a->compress->step = a->step;
    a->compress->keys = keys;
    a->compress->meta = meta;
    a->compress->n_bound = n_bound;
    a->compress->decode_follows = 1;
    a->compress->vals = vals;
    if (dense_vals) a->compress->dense_vals = dense_vals;   // one launch serves both kinds
    int rc = skml_compress_sparse(a->compress, stream);
    if (!rc && batch_keys) rc = batch_consumed(a, (cudaStream_t)stream);
    if (rc) return rc;
    a->decode->step = a->step;
    a->decode->lr = a->lr;
    a->decode->adam_scale = a->adam_scale;
    a->decode->loss_out = a->loss_out;
    return skml_decode_update(a->decode, stream);
}

extern "C" int skml_train_step(SkmlStepArgs* a, void* stream_) {
    if (!a || (!a->coded && (!a->compress || !a->decode))) return (int)cudaErrorInvalidValue;
    cudaStream_t stream = (cudaStream_t)stream_;
    double* const loss = a->partials_template + 3;   // (settled behind the gradient)
    if (a->t_colptr || a->tt_pair_ptr) {
        // transposed index: coefficients per row, then one gather-sum per distinct column
        int rc;
        if (a->tt_pair_ptr) {
            const cudaError_t e = cudaMemcpyAsync(a->partials, a->partials_template, 4 * sizeof(double), cudaMemcpyDeviceToDevice, stream);
            if (e != cudaSuccess) return (int)e;
            rc = skml_glm_coef(a->rowptr, a->cols, a->vals, a->labels, a->seg_lo[0], a->seg_cnt[0], a->nnz_padded,
                               a->avg_nnz, a->w, a->dim, (int)a->loss_id, (float)a->inv_batch, a->partials + 1, a->coef,
                               a->status, a->budget_cycles, stream_);
            if (rc) return rc;
            rc = skml_colsum_tiled(a->tt_tile_pair_ptr, a->tt_pair_ptr, a->tt_lrow, a->t_vals, a->tt_pair_dst, a->tt_col_pair_ptr,
                                   a->t_ucols, (int)a->tt_rows, (int)a->tt_tile_rows, (int)a->tt_tiles, (int)a->t_cols, a->coef,
                                   a->w, (float)a->lambda, a->tt_partial, a->gvals, stream_);
        } else {
            rc = skml_glm_coef_clear(a->rowptr, a->cols, a->vals, a->labels, a->seg_lo[0], a->seg_cnt[0], a->avg_nnz, a->w, a->dim,
                                     (int)a->loss_id, (float)a->inv_batch, loss, a->coef, a->gvals, a->t_long_col, (int)a->t_long,
                                     stream_);
            if (rc) return rc;
            if (a->hot_columns)
                rc = skml_hot_colsum(a->hot_columns, a->t_bins, (int)a->t_short, (int)a->t_medium, a->t_colptr, a->t_rowidx,
                                     a->t_vals, a->t_ucols, a->coef, a->w, (float)a->lambda, a->gvals, a->partials, a->partials_template, stream_);
            else
                rc = skml_colsum_settle(a->t_colptr, a->t_rowidx, a->t_vals, a->t_ucols, a->t_bins, a->t_long_col, a->t_long_e0,
                                        a->t_long_e1, (int)a->t_short, (int)a->t_medium, (int)a->t_long, a->coef, a->w,
                                        (float)a->lambda, a->gvals, a->partials, a->partials_template, stream_);
        }
        if (rc) return rc;
        rc = batch_consumed(a, stream);
        if (rc) return rc;
        return apply_gradient(a, a->t_ucols, a->t_meta, a->gvals, nullptr, a->t_cols, false, stream_);
    }
    if (a->l_ucols) {
        if (a->coded) return (int)cudaErrorInvalidValue;   // the sketch arm's alone
        const cudaError_t e = cudaMemcpyAsync(a->partials, a->partials_template, 4 * sizeof(double), cudaMemcpyDeviceToDevice, stream);
        if (e != cudaSuccess) return (int)e;
        // local-id batch: compact weights in, scatter into the compact accumulator, values out in key order
        const int n = (int)a->l_ncols;
        int rc = skml_gather_compact(a->w, a->l_ucols, n, a->wc, stream_);
        if (rc) return rc;
        for (int s = 0; s < 2; ++s) {
            if (a->seg_cnt[s] <= 0) continue;
            rc = skml_glm_grad(a->rowptr, a->cols, a->vals, a->labels, a->seg_lo[s], a->seg_cnt[s], a->nnz_padded,
                               a->avg_nnz, a->wc, a->gc, nullptr, (int)a->loss_id, (float)a->inv_batch, (int)a->hot,
                               a->partials + 1, a->status, a->budget_cycles, stream_);
            if (rc) return rc;
        }
        rc = skml_finalize_compact(a->gc, a->wc, (float)a->lambda, n, a->gvals, nullptr, stream_);  // no touched bitmap: every slot is a key
        if (rc) return rc;
        return apply_gradient(a, a->l_ucols, a->l_meta, a->gvals, nullptr, a->l_ncols, true, stream_);
    }
    if (a->dense_index) {
        int rc = skml_dt_gradient(a->dense_index, a->rowptr, a->cols, a->vals, a->labels, a->seg_lo[0], a->nnz_padded, a->avg_nnz, a->w,
                                  (int)a->loss_id, (float)a->inv_batch, loss, a->g, a->bitmap, a->status,
                                  a->budget_cycles, stream_);
        if (rc) return rc;
    }
    for (int s = 0; s < 2 && !a->dense_index; ++s) {
        if (a->seg_cnt[s] <= 0) continue;
        int rc = skml_glm_grad(a->rowptr, a->cols, a->vals, a->labels, a->seg_lo[s], a->seg_cnt[s], a->nnz_padded,
                               a->avg_nnz, a->w, a->g, a->bitmap, (int)a->loss_id, (float)a->inv_batch, (int)a->hot,
                               loss, a->status, a->budget_cycles, stream_);
        if (rc) return rc;
    }
    int rc = batch_consumed(a, stream);
    if (rc) return rc;
    rc = skml_compact_settle(a->g, a->w, a->bitmap, (int)a->dim, (float)a->lambda, a->block_counts, a->meta, a->keys,
                          a->gvals, a->dense_vals, a->n_max, a->status, a->partials, a->partials_template, stream_);
    if (rc) return rc;
    return apply_gradient(a, a->keys, a->meta, a->gvals, a->dense_vals, 0, false, stream_);
}
