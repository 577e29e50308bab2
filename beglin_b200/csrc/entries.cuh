// The entries that other files of the library call, beside their definitions: every file sees them, so that the compiler refuses a definition
// that has gone another way (with C linkage the linker would not notice).
#pragma once

extern "C" {
// attention.cu
int bg_attention_partial(const void* q, int q_dtype, int q_stride, const void* kv_pool, int cache_dtype, int num_pages, int page_size, const int* block_table,
    int max_pages, const int* positions, const int* qblk, int n_qblk, float* part_o, float* part_ml, int max_splits, int n_splits_launch, int nh, int nkv, int
    hd, int vd, int window, int split, int tile, int bq, float scale, float softcap, int keep, const float* slopes, int maps, unsigned* status, cudaStream_t
    stream);
int bg_attention_merge(const float* part_o, const float* part_ml, const int* positions, void* out, int out_dtype, int out_stride, int T, int nh, int hd, int
    max_splits, int split, int window, int sink, const float* sink_w, int keep, cudaStream_t stream);
// elementwise.cu
int bg_swiglu(const void* gu, int in_dtype, int parts, long long part_stride, void* out, int out_dtype, int rows, int im, int block, int act, float limit,
    cudaStream_t stream);
int bg_rope_kv_append(const void* src, int src_dtype, int src_stride, int parts, long long part_stride, void* q_out, int q_dtype, int q_stride, const float*
    cos_sin, const int* positions, const int* row_req, const int* block_table, int max_pages, void* kv_pool, int cache_dtype, int num_pages, int page_size,
    int T, int nh, int nkv, int hd, int rot, int interleaved, unsigned* status, cudaStream_t stream);
// gemm_f32.cu
long long bg_gemm_f32_scratch(int M, int N, int K, int batch);
int bg_gemm_f32_nt(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc, int M, int N, int K, int accumulate, float*
    scratch, unsigned* status, cudaStream_t stream);
// gemm_fused.cu
int bg_gemm_fused(const void* W, int n_out, int K, int ldw, const void* X, int ldx, const float* xf, int ldxf, const float* ssq_in, int n_ssq_in, int
    ssq_in_stride, const void* norm_w, float eps, int T, const float* bias, int mode, void* out, int out_dtype, int ldo, float* ssq_out, int ssq_out_stride,
    int splits, float limit, unsigned* status, cudaStream_t stream);
// gemm_grouped_pair.cu
int bg_gemm_grouped_pair(const void* W, int E, int n_out, int K, int ldw, const void* X, int rows, int ldx, void* out, int out_dtype, int ldo, const int*
    offsets, int act, unsigned* status, cudaStream_t stream);
// gemm_grouped_tc.cu
int bg_gemm_grouped_tc(const void* W, int E, int n_out, int K, int ldw, const void* X, int rows, int ldx, void* out, int out_dtype, int ldo, const int*
    offsets, int act, unsigned* status, cudaStream_t stream);
// gemm_heads.cu
int bg_gemm_heads(const void* W, int H, int n_out, int K, const void* X, long long x_rows, int x_cols, int ldx, int x_row, int x_col, int T, void* out, int
    out_dtype, long long out_head, int out_row, const void* gate, int gate_dtype, int gate_stride, int gate_col, int per_feature, unsigned* status,
    cudaStream_t stream);
// gemm_tcgen05.cu
int bg_gemm_bf16_tn(const void* W, int n_out, int K, int ldw, const void* X, int T, int ldx, const float* bias, void* out, int out_dtype, int ldo, int splits,
    unsigned* status, cudaStream_t stream);
// latent_attention.cu
int bg_latent_append(const void* src, int src_dtype, int src_stride, int col0, int rank, int rot, int rot_dims, const void* w, int w_dtype, float eps, const
    float* cos_sin, const int* positions, const int* row_req, const int* block_table, int max_pages, void* pool, int pool_dtype, int num_pages, int page_size,
    int n_rows, unsigned* status, int q_col0, int q_rank, const void* q_w, void* q_out, int q_dtype, cudaStream_t stream);
int bg_latent_attention_merge(const float* part_o, const float* part_ml, const int* positions, void* out, int out_dtype, long long out_head, int out_row, int
    T, int H, int rank, int max_splits, int split, int window, const float* sink_w, int ctas, cudaStream_t stream);
// latent_attention_mma.cu
int bg_latent_attention_mma_partial(const float* q_lat, long long ql_head, int ql_row, const void* q_raw, int qr_row, int qr_head, int qr_off, const float*
    cos_sin, const void* pool, int num_pages, int page_size, const int* block_table, int max_pages, const int* positions, const int* qblk, int n_qblk, float*
    part_o, float* part_ml, int max_splits, int n_splits_launch, int H, int hc, int rank, int rot, int rot_dims, int split, int bq, int stages, int window,
    float scale, unsigned* status, cudaStream_t stream);
// latent_attention_tcgen05.cu
int bg_latent_attention_tc_partial(const float* q_lat, long long ql_head, int ql_row, const void* q_raw, int qr_row, int qr_head, int qr_off, const float*
    cos_sin, const void* pool, int num_pages, int page_size, const int* block_table, int max_pages, const int* positions, const int* qblk, int n_qblk, float*
    part_o, float* part_ml, int max_splits, int H, int rank, int rot, int rot_dims, int window, float scale, unsigned* status, cudaStream_t stream);
// mamba2.cu
int bg_conv_silu(const void* src, int src_dtype, int src_stride, int col0, int channels, int taps, const void* w, const void* b, int w_dtype, float* state,
    long long slot_stride, long long conv_off, const int* slots, const int* row_req, const int* reqs, int n_req, float* out, int n_rows, int act, const float*
    src_bias, int* launched, cudaStream_t stream);
int bg_ssm_scan(const float* xbc, int channels, const void* src, int src_dtype, int src_stride, int dt_col, const void* dt_bias, const void* A_log, const
    void* D, int w_dtype, float* state, long long slot_stride, const int* slots, const int* reqs, int n_req, float* y, int H, int P, int N, int G,
    cudaStream_t stream);
int bg_gated_group_rmsnorm(const float* y, const void* src, int src_dtype, int src_stride, int z_col, const void* w, int w_dtype, float eps, void* out, int
    out_dtype, int n_rows, int inner, int groups, int mode, cudaStream_t stream);
// mamba2_chunked.cu
int bg_ssm_chunked(const float* xbc, int channels, const void* src, int src_dtype, int src_stride, int dt_col, const void* dt_bias, const void* A_log, const
    void* D, int w_dtype, float* state, long long slot_stride, const int* slots, const int* chunks, int n_chunks, const int* longs, int n_long, float* scores,
    float* work, float* decay, float* y, int H, int P, int N, int G, int tensor_cores, unsigned* status, cudaStream_t stream);
// moe.cu
int bg_route_layout_counts(int T, int d, int E, int top);
int bg_route_layout_wins(int T, int d, int E, int top);
int bg_route_rows_takes(int T, int d, int E, int top);
int bg_route_place(const void* h, int h_dtype, int ldh, const float* W, int T, int d, int E, int top, int mode, int renorm, const float* bias, float scale,
    const float* logit_bias, int* ids, float* weights, int* offsets, int* row_of, int* src_of, void* xp, int scale_input, int* hist, int n_hist, int*
    launched, cudaStream_t stream);
int bg_route_combine(const void* yp, int y_dtype, const float* weights, const int* row_of, float* out, int T, int d, int top, int scale, cudaStream_t stream);
int bg_route_combine_ext(const void* yp, int y_dtype, const float* weights, const int* row_of, const int* ids, int n_real, const void* h, int h_dtype, int
    ldh, const float* shared, const void* sg, int sg_dtype, int sg_stride, float* out, int T, int d, int top, cudaStream_t stream);
int bg_glu_clamped(const void* gu, int gu_dtype, int ld, void* out, int out_dtype, int rows, int n, float limit, float alpha, cudaStream_t stream);
// rglru.cu
int bg_rglru_split(const float* u, void* x2, int T, int W, int blocks, cudaStream_t stream);
// sampling.cu
long long bg_sample_scratch_bytes(int n);
int bg_sample(const float* logits, int n, int V, const float* temperature, const float* uniform, int* out, void* scratch, cudaStream_t stream);
}
