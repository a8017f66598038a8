/*
 * nb_encoder.h -- C ABI of the token-wise kernels around attention in the packed inference encoder
 * (nanobrain_b200.model.ViTMAE3D.embed_packed): selecting in-mask patches, gathering them, adding
 * position embeddings and class tokens, residual + LayerNorm, GELU, and the final norm with its mean and
 * dense grid. The arithmetic is that of the modules under bf16 autocast (src/nanobrain/modules.py:68-131
 * and src/nanobrain/model.py:124-141, 254-285): fp32 residual stream and LayerNorm, bf16 operands of the
 * Linears.
 *
 * Conventions as in nb_attn.h: device pointers unless said otherwise, asynchronous on `stream`, nothing
 * is allocated and nothing kept. Return values are enum nb_attn_error codes. Rows are contiguous; `dim`
 * is a multiple of 64, at most NB_ENC_MAX_DIM; pointers are 16-byte aligned.
 */
#ifndef NB_ENCODER_H_
#define NB_ENCODER_H_

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

#define NB_ENC_MAX_DIM 1024
#define NB_ENC_MAX_IMAGES 64 /* per call; callers with more images make several calls */

typedef struct nb_enc_cast_item {
  const float* src;
  void* dst; /* bf16 */
  int64_t n; /* elements */
} nb_enc_cast_item;

/* dst = bf16(src) for every item (`items` is a host array). */
int nb_enc_cast(const nb_enc_cast_item* items, int n_items, void* stream);

/* For images [first, first + n): the in-mask patches in ascending order. masks: host array of n device
 * pointers to `patches` bytes each (0 / 1). ids, rank: [images][patches]; ids[i][j] = patch of the j-th
 * in-mask one, rank[i][p] = its position or -1. counts: [images]. */
int nb_enc_select(const uint8_t* const* masks, int first, int n, int patches, int32_t* ids, int32_t* rank,
                  int32_t* counts, void* stream);

/* cu[i] = tokens before image i, cu_r[i] = the same with `class_tokens` rows per image before its tokens
 * (both [images + 1]); host_counts (pinned host memory) receives the counts. */
int nb_enc_offsets(const int32_t* counts, int images, int class_tokens, int32_t* cu, int32_t* cu_r,
                   int32_t* host_counts, void* stream);

/* tokens[cu[i] + j] = bf16(values[i][ids[i][j]]), `dim` values per patch (any multiple of 4). values:
 * host array of n device pointers to fp32 [patches][dim]. */
int nb_enc_gather(const float* const* values, int first, int n, int patches, int dim, const int32_t* ids,
                  const int32_t* counts, const int32_t* cu, void* tokens, void* stream);

/* One LayerNorm: y = (x - mean) / sqrt(var + eps) * gamma + beta over `dim`, fp32. */
typedef struct nb_enc_norm {
  const float* gamma;
  const float* beta;
  float eps;
} nb_enc_norm;

/* x (fp32 [rows][dim]) = class tokens and h + position embeddings (three tables indexed by the patch's
 * coordinate, coord: int64 [patches][3]); y (bf16) = norm(x). rows = cu_r[images]. */
int nb_enc_embed(const void* h, const int32_t* ids, const int32_t* cu, const int32_t* cu_r, int images, int patches,
                 int class_tokens, int64_t rows, int dim, const int64_t* coord, const float* table_x,
                 const float* table_y, const float* table_z, const float* cls, float* x, const nb_enc_norm* norm,
                 void* y, void* stream);

/* x += add (bf16); y (bf16) = norm(x). */
int nb_enc_add_norm(float* x, const void* add, int64_t rows, int dim, const nb_enc_norm* norm, void* y, void* stream);

/* v = gelu(v), exact (erf), bf16 in place; n a multiple of 8. */
int nb_enc_gelu(void* v, int64_t n, void* stream);

/* y = norm(x + add) in fp32 for the patch tokens of images [first, first + n): dense (host array of n device
 * pointers to fp32 [patches][dim], or NULL) receives y at the patch's place and 0 outside the mask, means
 * [images][dim] the mean of y over the image's patches. scratch: nb_enc_finish_scratch_bytes(n, patches, dim). */
int nb_enc_finish(const float* x, const void* add, const int32_t* rank, const int32_t* counts, const int32_t* cu_r,
                  int first, int n, int patches, int class_tokens, int dim, const nb_enc_norm* norm,
                  float* const* dense, float* means, void* scratch, void* stream);
size_t nb_enc_finish_scratch_bytes(int n, int patches, int dim);

#ifdef __cplusplus
}
#endif
#endif /* NB_ENCODER_H_ */
