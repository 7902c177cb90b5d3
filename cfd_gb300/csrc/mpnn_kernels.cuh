// mpnn_kernels.cuh — declarations of the kernels in kernels_mpnn.cu.
#pragma once
#include "mpnn.cuh"

namespace cfd {
namespace mpnn {

// row chunks of the weight gradients: one block per SM of the 152
constexpr int kTrainChunks = 152;

// kernels with a `gate` argument return at once when gate != null and *gate == 0
__global__ void k_globals(int nb, const int* bnode, const int* bkind, const double* gx,
                          const double* gy, const double* X, const double* Y, Globals* G,
                          const int* gate);
__global__ void k_scatter_bc(int nb, const int* bnode, const double* gx, const double* gy,
                             double* gnx, double* gny, const int* gate);
__global__ void k_fields_seed(int n, const float* y, const int* kind, const Globals* G, double* F);
__global__ void k_fields_guess(int n, const int* kind, const Globals* G, const double* F,
                               const double* x0, const double* x1, double* c0, double* c1,
                               float2* s0, float2* s1);
__global__ void k_fields_update(int n, const int* kind, const Globals* G, const double* x0,
                                const double* x1, double* F);
__global__ void k_features(int n, const double* X, const double* Y, const int* kind,
                           const Globals* G, float* f, const int* gate);
__global__ void k_edge_features(int m, const int* src, const int* nbr, const double* X,
                                const double* Y, const Globals* G, float* e, const int* gate);
// FP32 training passes (kernels_mpnn.cu): P|Q = [A; B] h; v = U [h; agg] + u and h1 = h +
// relu(v), from the transposed weights that k_encode leaves in wt; their backward products
// (dhc = [dh | dagg / deg], dh += its first half + dPQ [A; B])
int dense_pq(cudaStream_t st, int n, const float* h, const float* W, float* pq);
int dense_update(cudaStream_t st, int n, const float* h, const float* agg, const float* W,
                 const float* b, float* v, float* h1);
int dense_update_bwd(cudaStream_t st, int n, const float* dh, const float* v, const float* W,
                     const int* ptr, float* dhc);
int dense_pq_bwd(cudaStream_t st, int n, const float* dpq, const float* W, const float* dhc,
                 float* dh);
// weight gradients of layer `layer` into the chunk rows of part
int wgrad_update(cudaStream_t st, int n, const float* dh, const float* v, const float* h,
                 const float* agg, float* part, int layer);
int wgrad_pq(cudaStream_t st, int n, const float* dpq, const float* h, float* part, int layer);
constexpr unsigned kEdgeBlocks = 152 * 6;  // blocks of k_edge_fwd at most (resident)
constexpr int kEncodeExtra = 64;  // blocks of k_encode that transpose the weights
__global__ void k_encode(int n, const float* f, const float* w, float* h, float* wt);
__global__ void k_wgrad_in(int n, const float* dh, const float* h0, const float* f, float* part);
__global__ void k_fold(int nq, const float* part, float* out, float* loss);
__global__ void k_edge_fwd(int n, const int* ptr, const int* nbr, const float* PQ, const float* e,
                           const float* C, const float* c, ushort4* mask, float* agg);
__global__ void k_edge_bwd(int n, const int* ptr, const int* nbr, const int* rev,
                           const ushort4* mask, const float* dhc, const float* e, float* dPQ,
                           float* part, int off);
__global__ void k_decode(int n, const float* h, const float* w, float* y, const float* target,
                         const int* kind, float inv_nfree, float* dh, float* part);
__global__ void k_adam(int np, float* w, const float* g, float* m, float* v, float lr, float b1,
                       float b2, float eps, float bc1, float bc2);
__global__ void k_targets(int n, const double* phi, const double* psx, const double* psy,
                          const Globals* G, float* t);
__global__ void k_guess(int n, const float* y, const int* kind, const double* gnx,
                        const double* gny, const Globals* G, double* ux, double* uy,
                        const int* gate);

// BF16 tensor-core inference: y[n][OUT] from the features; wb (BF16 copy of w) is refreshed
// when *wb_valid is false
int infer_bf16(cudaStream_t st, const float* w, __nv_bfloat16* wb, bool* wb_valid, int n,
               const int* ptr, const int* nbr, const float* f, const float* e,
               __nv_bfloat16* hb, __nv_bfloat16* pqb, float* y, const int* gate, int* err);

}  // namespace mpnn
}  // namespace cfd
