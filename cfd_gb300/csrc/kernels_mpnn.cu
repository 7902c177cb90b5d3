// kernels_mpnn.cu — kernels of the learned mesh-motion guess (mpnn.cuh): boundary
// statistics and features, the FP32 training forward and backward passes, Adam, and the
// BF16 tensor-core inference pass.
//
// Graph arrays: ptr/nbr = CSR point neighbours (0-based, symmetric); src[k] = the source
// node of edge k = (src[k] -> nbr[k]); rev[k] = the index of the reverse edge.
// Reductions over nodes or edges (weight gradients, loss) go through per-block partials
// folded in a fixed order, so a training step is deterministic.
#include <algorithm>
#include <type_traits>

#include "mpnn_kernels.cuh"

namespace cfd {
namespace mpnn {

static_assert((N_PARAMS + 1) % 4 == 0 && L_SIZE % 4 == 0 && LAYER0 % 4 == 0 && L_U % 4 == 0,
              "float4 accesses to the weights and to the rows of the partial gradients");

// ------------------------------------------------------------------ globals and features
// One block of 256 threads.  Boundary nodes are listed in bnode[0..nb) with their kind and
// prescribed displacement (gx, gy).  Body geometry (c, L, R) and the least-squares affine
// fit g = t + M d, d = p - c, over the body nodes: since sum d = 0, t = mean g and each row
// of M solves [Sxx Sxy; Sxy Syy] m = [sum g d_x; sum g d_y].  A launch is latency: a
// dependent FP64 add waits 64 clocks, so the sums of a pass are formed side by side
// (block_trees) and a thread's nodes are loaded four at a time (34 us beside a 262,144-node step
// with one tree after the other, 21 us now).
__global__ void k_globals(int nb, const int* __restrict__ bnode, const int* __restrict__ bkind,
                          const double* __restrict__ gx, const double* __restrict__ gy,
                          const double* __restrict__ X, const double* __restrict__ Y,
                          Globals* __restrict__ G, const int* __restrict__ gate) {
    if (gate && !*gate) return;
    __shared__ double sh[9][kTreePad], out[9];
    __shared__ double rmax_s;
    const int t = threadIdx.x;
    constexpr int B = 4;
    double a[6] = {};  // body nodes, sum x, sum y, sum gx, sum gy, outer nodes
    for (int k0 = t; k0 < nb; k0 += 256 * B) {
        int kd[B], p[B];
        double x[B], y[B], u[B], v[B];
#pragma unroll
        for (int q = 0; q < B; ++q) {
            const int k = min(k0 + 256 * q, nb - 1);
            p[q] = bnode[k];
            kd[q] = bkind[k];
            u[q] = gx[k];
            v[q] = gy[k];
        }
#pragma unroll
        for (int q = 0; q < B; ++q) {
            x[q] = X[p[q]];
            y[q] = Y[p[q]];
        }
#pragma unroll
        for (int q = 0; q < B; ++q) {
            if (k0 + 256 * q >= nb) break;
            if (kd[q] == KIND_BODY) {
                a[0] += 1.0;
                a[1] += x[q];
                a[2] += y[q];
                a[3] += u[q];
                a[4] += v[q];
            } else {
                a[5] += 1.0;
            }
        }
    }
    block_trees(a, sh, out);
    const double nbody = out[0], nout = out[5];
    const double inb = nbody > 0 ? 1.0 / nbody : 0.0;
    const double cx = out[1] * inb, cy = out[2] * inb, sgx = out[3], sgy = out[4];
    __syncthreads();  // out is written again
    double rmax = 0, s[8] = {};  // sum r (outer), Sxx, Sxy, Syy, sums of g d
    for (int k0 = t; k0 < nb; k0 += 256 * B) {
        int kd[B], p[B];
        double x[B], y[B], u[B], v[B];
#pragma unroll
        for (int q = 0; q < B; ++q) {
            const int k = min(k0 + 256 * q, nb - 1);
            p[q] = bnode[k];
            kd[q] = bkind[k];
            u[q] = gx[k];
            v[q] = gy[k];
        }
#pragma unroll
        for (int q = 0; q < B; ++q) {
            x[q] = X[p[q]];
            y[q] = Y[p[q]];
        }
#pragma unroll
        for (int q = 0; q < B; ++q) {
            if (k0 + 256 * q >= nb) break;
            const double dx = x[q] - cx, dy = y[q] - cy;
            const double r = sqrt(dx * dx + dy * dy);
            if (kd[q] == KIND_BODY) {
                rmax = fmax(rmax, r);
                s[1] += dx * dx;
                s[2] += dx * dy;
                s[3] += dy * dy;
                s[4] += u[q] * dx;
                s[5] += u[q] * dy;
                s[6] += v[q] * dx;
                s[7] += v[q] * dy;
            } else {
                s[0] += r;
            }
        }
    }
    sh[8][t] = rmax;
    block_trees(s, sh, out);
    if (t < 32) {
        double m = sh[8][t];
#pragma unroll
        for (int q = 1; q < 8; ++q) m = fmax(m, sh[8][t + 32 * q]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
        if (t == 0) rmax_s = m;
    }
    __syncthreads();
    if (t == 0) {
        const double rmax = rmax_s, rsum = out[0], sxx = out[1], sxy = out[2], syy = out[3];
        const double gxdx = out[4], gxdy = out[5], gydx = out[6], gydy = out[7];
        Globals g;
        g.cx = cx;
        g.cy = cy;
        g.L = rmax > 0 ? 2.0 * rmax : 1.0;
        g.R = nout > 0 ? rsum / nout : g.L;
        g.tx = sgx * inb;
        g.ty = sgy * inb;
        const double det = sxx * syy - sxy * sxy;
        const double id = det > 0 ? 1.0 / det : 0.0;
        g.m11 = (syy * gxdx - sxy * gxdy) * id;
        g.m12 = (sxx * gxdy - sxy * gxdx) * id;
        g.m21 = (syy * gydx - sxy * gydy) * id;
        g.m22 = (sxx * gydy - sxy * gydx) * id;
        // second-moment ellipse: eigenvalues of [sxx sxy; sxy syy] / nbody
        const double hx = 0.5 * (sxx - syy) * inb, mxy = sxy * inb, tr = 0.5 * (sxx + syy) * inb;
        const double rt = sqrt(hx * hx + mxy * mxy);
        g.ea = sqrt(2.0 * (tr + rt));
        g.eb = sqrt(fmax(2.0 * (tr - rt), 0.0));
        const double al = 0.5 * atan2(2.0 * mxy, 2.0 * hx);
        g.ec = cos(al);
        g.es = sin(al);
        const double a[2][3] = {{g.tx, g.m11, g.m12}, {g.ty, g.m21, g.m22}};
        double iq[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double q = a[s][0] * a[s][0] + a[s][1] * a[s][1] + a[s][2] * a[s][2];
            iq[s] = q > 0.0 ? 1.0 / q : 0.0;
        }
        g.iqx = iq[0];
        g.iqy = iq[1];
        *G = g;
    }
}

// Basis fields kept per node in FP64 (planes F[0..2] = Phi, Psi_x, Psi_y in length units)
// for the refined learned guess: seeded from a network run, combined with each solve's
// affine fit (G) into its guess, and corrected by each solve's solution.
// Seed: F = (y0, L y1, L y2) at the free nodes, 0 elsewhere.
__global__ void k_fields_seed(int n, const float* __restrict__ y, const int* __restrict__ kind,
                              const Globals* __restrict__ G, double* __restrict__ F) {
    const double L = G->L;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const bool f = kind[i] == KIND_FREE;
        F[i] = f ? (double)y[OUT * i] : 0.0;
        F[n + i] = f ? L * (double)y[OUT * i + 1] : 0.0;
        F[2 * (size_t)n + i] = f ? L * (double)y[OUT * i + 2] : 0.0;
    }
}

// Guess: c = t Phi + M (Psi_x, Psi_y) at the free nodes (x: (tx, m11, m12), y: (ty, m21,
// m22)); the boundary nodes keep x, which already holds this solve's Dirichlet values.
__global__ void k_fields_guess(int n, const int* __restrict__ kind, const Globals* __restrict__ G,
                               const double* __restrict__ F, const double* __restrict__ x0,
                               const double* __restrict__ x1, double* __restrict__ c0,
                               double* __restrict__ c1, float2* __restrict__ s0,
                               float2* __restrict__ s1) {
    const Globals g = *G;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double a = x0[i], b = x1[i];
        if (kind[i] == KIND_FREE) {
            const double f0 = F[i], f1 = F[n + i], f2 = F[2 * (size_t)n + i];
            a = g.tx * f0 + g.m11 * f1 + g.m12 * f2;
            b = g.ty * f0 + g.m21 * f1 + g.m22 * f2;
        }
        c0[i] = a;
        c1[i] = b;
        if (s0) {  // relative tests: hi + lo, the precise product's operand
            float hi, lo;
            split_bits(a, hi, lo);
            s0[i] = make_float2(hi, lo);
            split_bits(b, hi, lo);
            s1[i] = make_float2(hi, lo);
        }
    }
}

// Correction after the solves: each solve s with coefficients a_s (its affine fit) and
// solution x_s gives one equation a_s . F_i = x_s(i) per node; F_i moves to the nearest
// point that satisfies it (a Kaczmarz step per node: the x solve's, then the y solve's;
// solves with no prescribed motion are skipped).
__global__ void k_fields_update(int n, const int* __restrict__ kind, const Globals* __restrict__ G,
                                const double* __restrict__ x0, const double* __restrict__ x1,
                                double* __restrict__ F) {
    const Globals g = *G;
    const double a[2][3] = {{g.tx, g.m11, g.m12}, {g.ty, g.m21, g.m22}};
    const double iq[2] = {g.iqx, g.iqy};  // formed once, with the fit
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (kind[i] != KIND_FREE) continue;
        double f[3] = {F[i], F[n + i], F[2 * (size_t)n + i]};
        const double x[2] = {x0[i], x1[i]};
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            if (iq[s] == 0.0) continue;
            const double r = (x[s] - (a[s][0] * f[0] + a[s][1] * f[1] + a[s][2] * f[2])) * iq[s];
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c] += a[s][c] * r;
        }
        F[i] = f[0];
        F[n + i] = f[1];
        F[2 * (size_t)n + i] = f[2];
    }
}

// per-node prescribed displacement (0 at free nodes) from the boundary list
__global__ void k_scatter_bc(int nb, const int* __restrict__ bnode, const double* __restrict__ gx,
                             const double* __restrict__ gy, double* __restrict__ gnx,
                             double* __restrict__ gny, const int* __restrict__ gate) {
    if (gate && !*gate) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nb) return;
    gnx[bnode[k]] = gx[k];
    gny[bnode[k]] = gy[k];
}

// Geometry-only node features: position, log-radius, boundary kinds, and the three fields
// of a continuum model of the mesh-motion operator, which the network corrects.  The
// operator's entries grad N_i . grad N_j q carry no area factor (mLaplace.f90:40, 48), so in
// the continuum it is div(k grad u) with k ~ 1/(element area), k ~ 1/r^2 on O-grids whose
// spacing grows with r.  For a circular body of radius a = L/2 inside a circle of radius R:
// Phi = (R^2 - r^2)/(R^2 - a^2) (clamped to [0, 1]) and Psi = psi(rho) d / rho with
// psi(r) = a ((r/R)^p - (r/R)^q) / ((a/R)^p - (a/R)^q), p, q = 1 +- sqrt(2), over L, where
// rho = r a / r_b(theta) stretches the body's second-moment ellipse (radius r_b along the
// node's direction) onto the circle of radius a, so that Psi = d on the body.  Feature 9 is
// the ellipse's aspect ratio.
__global__ void k_features(int n, const double* __restrict__ X, const double* __restrict__ Y,
                           const int* __restrict__ kind, const Globals* __restrict__ G,
                           float* __restrict__ f, const int* __restrict__ gate) {
    if (gate && !*gate) return;
    // per-graph constants (FP32 arithmetic below; positions are differenced in FP64)
    const Globals g = *G;
    const float L = (float)g.L, iL = 1.f / L, a = 0.5f * L, R = (float)g.R;
    const float ea = (float)g.ea, eb = (float)g.eb, ec = (float)g.ec, es = (float)g.es;
    const float p = 2.41421356f, q = -0.41421356f;
    const float ar = a / R, den = powf(ar, p) - powf(ar, q);
    const float logRL = logf(R * iL), aspect = ea > 0.f ? eb / ea : 1.f;
    const bool annulus = R > a;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float dx = (float)(X[i] - g.cx), dy = (float)(Y[i] - g.cy);
        const float r2 = dx * dx + dy * dy, r = sqrtf(r2);
        float* o = f + (size_t)i * F_IN;
        o[0] = dx * iL;
        o[1] = dy * iL;
        o[2] = logf(r * iL + 1e-6f);
        o[3] = logRL;
        o[4] = kind[i] == KIND_BODY ? 1.f : 0.f;
        o[5] = kind[i] == KIND_OUTER ? 1.f : 0.f;
        float phi = 0.f, c = 0.f;
        if (annulus && r < R) {
            phi = (R * R - r2) / (R * R - a * a);
            const float rs = fmaxf(r, 1e-6f * L);
            // body radius along the node's direction (frame of the ellipse's axes)
            const float u = (dx * ec + dy * es) / rs, v = (-dx * es + dy * ec) / rs;
            const float rb = ea * eb / fmaxf(sqrtf(eb * eb * u * u + ea * ea * v * v), 1e-30f);
            const float rho = fminf(rs * a / fmaxf(rb, 1e-6f * L), 0.999999f * R);
            const float rr = rho / R;
            c = a * (powf(rr, p) - powf(rr, q)) / den / rho;
        }
        o[6] = fminf(fmaxf(phi, 0.f), 1.f);
        o[7] = c * dx * iL;
        o[8] = c * dy * iL;
        o[9] = aspect;
    }
}

__global__ void k_edge_features(int m, const int* __restrict__ src, const int* __restrict__ nbr,
                                const double* __restrict__ X, const double* __restrict__ Y,
                                const Globals* __restrict__ G, float* __restrict__ e,
                                const int* __restrict__ gate) {
    if (gate && !*gate) return;
    const float iL = (float)(1.0 / G->L);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        const int i = src[k], j = nbr[k];
        const float dx = (float)(X[j] - X[i]), dy = (float)(Y[j] - Y[i]);
        const float ln = sqrtf(dx * dx + dy * dy), il = 1.f / ln;
        e[3 * (size_t)k] = dx * il;
        e[3 * (size_t)k + 1] = dy * il;
        e[3 * (size_t)k + 2] = logf(ln * iL);
    }
}

// ------------------------------------------------------------------ FP32 training passes
// The ~40 kernels of a loss and gradient run one after the other in one stream, 10 to 35 us each
// at 49,794 nodes, and are launched as a chain (launch_chain): a kernel's blocks are placed while
// the one ahead drains, 1.00 -> 0.92 ms of a pass.

// ------------------------------------------------------------------ FP32 dense layers
// The dense products of a training step, n x 64 or n x 128 rows against 64 x 128 weights: a
// register-tiled FP32 GEMM, bound by the FP32 pipe.  A block holds the whole weight matrix in
// shared memory as [k][column]; each of its warps walks over row groups of its own (16 rows,
// private to the warp, so that no block barrier separates one warp's loads from another's
// FMAs).  A thread forms 8 rows x 8 columns (N = 128; 24 shared wavefronts for 256 FMAs of a
// step of four k) or 4 x 8 (N = 64).  The lanes of a warp that share columns take adjacent
// rows of a 4-float padded tile, and a thread's columns come in two groups of four, which
// keeps every vector load free of bank conflicts.  Each output sums its k in ascending order
// from the bias.  49,794 nodes: 112-154 us per product with one output column and 32 rows
// per thread and the weights re-read from global memory, 35-45 us with 8 x 4 outputs in
// 64-row block tiles, 28-33 us now.
constexpr int GR = 16;  // rows of a warp's group
// what the product's epilogue does
enum : int {
    GE_PLAIN = 0,     // Y = acc
    GE_RESIDUAL = 1,  // Y = acc (v), Y2 = X + relu(acc) with X the first 64 columns of the input
    GE_SPLIT = 2,     // columns 64.. divided by the node's degree: [d h | d agg / deg]
    GE_ACCUM = 3      // Y = (Y + E) + acc, E the first 64 columns of a 128-wide row
};
template <int K, int N>
struct GemmShape {
    static constexpr int RT = N / 16;              // rows per thread
    static constexpr int RG = GR / RT;             // row groups of a warp (2 or 4)
    static constexpr int L = 32 / RG;              // lanes over the columns
    static constexpr int KS = K + 4;               // padded row stride
    static constexpr int WARPS = N == 128 ? 8 : 16;
    static constexpr int PER_SM = N == 128 ? 2 : 1;
    static constexpr int SMEM = 4 * (K * N + WARPS * GR * KS);
    static_assert(8 * L == N && RT * RG == GR, "thread tile");
};

// Y[n][N] = X[n][K] . W[K][N].  The weights come by cp.async while the warp loads its first rows.  X is
// [X1 | X2] in 64-column halves when X2 is given (K = 128), and masked (X1 where gate > 0,
// else 0) when gate is given.
template <int K, int N, int EPI>
__global__ void __launch_bounds__(32 * GemmShape<K, N>::WARPS, GemmShape<K, N>::PER_SM)
k_gemm(int n, const float* __restrict__ X1, const float* __restrict__ X2,
       const float* __restrict__ gate, const float* __restrict__ W, const float* __restrict__ bias,
       const int* __restrict__ ptr, const float* __restrict__ E, float* __restrict__ Y,
       float* __restrict__ Y2) {
    typedef GemmShape<K, N> G;
    extern __shared__ __align__(16) float gsm[];
    float* Bs = gsm;  // K x N
    constexpr int T = 32 * G::WARPS, RT = G::RT, KS = G::KS;
    const int tid = threadIdx.x, lane = tid & 31;
    float* Xs = gsm + K * N + (tid >> 5) * GR * KS;  // the warp's rows
    const int z = chain_wait();
    W += z;
    const unsigned bs = (unsigned)__cvta_generic_to_shared(Bs);
#pragma unroll
    for (int q = tid; q < K * N / 4; q += T)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(bs + 16 * q), "l"(W + 4 * q)
                     : "memory");
    const int c0 = 4 * (lane % G::L), c1 = c0 + N / 2, rg = lane / G::L;
    float4 ba = make_float4(0.f, 0.f, 0.f, 0.f), bb = ba;
    if (bias) {
        ba = *reinterpret_cast<const float4*>(bias + c0);
        bb = *reinterpret_cast<const float4*>(bias + c1);
    }
    const int ngroup = (n + GR - 1) / GR;
    // each warp comes here once, before its first rows' products: a barrier of its own
    auto weights_ready = [&]() {
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");
    };
    bool ready = false;
    // groups interleaved over the blocks, so that a last partial round spreads over all SMs
    for (int grp = (tid >> 5) * gridDim.x + blockIdx.x; grp < ngroup; grp += gridDim.x * G::WARPS) {
        const int base = grp * GR + z;
        __syncwarp();  // the previous group has been read
#pragma unroll 16
        for (int q = lane; q < GR * K / 4; q += 32) {
            const int r = q / (K / 4), k = 4 * (q - r * (K / 4)), row = base + r;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < n) {
                // one address, not a load on either side of a branch: a group's loads go out together
                const float* src = K == 128 && X2 ? (k < 64 ? X1 : X2 - 64) + (size_t)row * 64 + k
                                                  : X1 + (size_t)row * K + k;
                v = *reinterpret_cast<const float4*>(src);
                if (gate) {
                    const float4 g = *reinterpret_cast<const float4*>(gate + (size_t)row * K + k);
                    v = make_float4(g.x > 0.f ? v.x : 0.f, g.y > 0.f ? v.y : 0.f,
                                    g.z > 0.f ? v.z : 0.f, g.w > 0.f ? v.w : 0.f);
                }
            }
            *reinterpret_cast<float4*>(Xs + r * KS + k) = v;
        }
        if (!ready) {
            weights_ready();
            ready = true;
        }
        __syncwarp();
        float acc[RT][8];
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            acc[i][0] = ba.x;
            acc[i][1] = ba.y;
            acc[i][2] = ba.z;
            acc[i][3] = ba.w;
            acc[i][4] = bb.x;
            acc[i][5] = bb.y;
            acc[i][6] = bb.z;
            acc[i][7] = bb.w;
        }
#pragma unroll 1
        for (int k = 0; k < K; k += 4) {
            float4 x[RT];
#pragma unroll
            for (int i = 0; i < RT; ++i)
                x[i] = *reinterpret_cast<const float4*>(Xs + (G::RG * i + rg) * KS + k);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 b0 = *reinterpret_cast<const float4*>(Bs + (k + u) * N + c0);
                const float4 b1 = *reinterpret_cast<const float4*>(Bs + (k + u) * N + c1);
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    const float xv = u == 0 ? x[i].x : u == 1 ? x[i].y : u == 2 ? x[i].z : x[i].w;
                    acc[i][0] = fmaf(xv, b0.x, acc[i][0]);
                    acc[i][1] = fmaf(xv, b0.y, acc[i][1]);
                    acc[i][2] = fmaf(xv, b0.z, acc[i][2]);
                    acc[i][3] = fmaf(xv, b0.w, acc[i][3]);
                    acc[i][4] = fmaf(xv, b1.x, acc[i][4]);
                    acc[i][5] = fmaf(xv, b1.y, acc[i][5]);
                    acc[i][6] = fmaf(xv, b1.z, acc[i][6]);
                    acc[i][7] = fmaf(xv, b1.w, acc[i][7]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            const int r = G::RG * i + rg, row = base + r;
            if (row >= n) break;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = h ? c1 : c0;
                float4 o = make_float4(acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2],
                                       acc[i][4 * h + 3]);
                float4* y = reinterpret_cast<float4*>(Y + (size_t)row * N + c);
                if (EPI == GE_RESIDUAL) {
                    const float4 x = *reinterpret_cast<const float4*>(Xs + r * KS + c);
                    *reinterpret_cast<float4*>(Y2 + (size_t)row * N + c) =
                        make_float4(x.x + fmaxf(o.x, 0.f), x.y + fmaxf(o.y, 0.f),
                                    x.z + fmaxf(o.z, 0.f), x.w + fmaxf(o.w, 0.f));
                } else if (EPI == GE_SPLIT) {
                    if (h) {
                        const float deg = (float)max(ptr[row + 1] - ptr[row], 1);
                        o = make_float4(o.x / deg, o.y / deg, o.z / deg, o.w / deg);
                    }
                } else if (EPI == GE_ACCUM) {
                    const float4 d = *y;
                    const float4 e = *reinterpret_cast<const float4*>(E + (size_t)row * 128 + c);
                    o = make_float4((d.x + e.x) + o.x, (d.y + e.y) + o.y, (d.z + e.z) + o.z,
                                    (d.w + e.w) + o.w);
                }
                *y = o;
            }
        }
    }
    if (!ready) weights_ready();  // a warp without rows
}

template <int K, int N, int EPI>
static int gemm(cudaStream_t st, int n, const float* X1, const float* X2, const float* gate,
                const float* W, const float* bias, const int* ptr, const float* E, float* Y,
                float* Y2) {
    typedef GemmShape<K, N> G;
    // the attribute belongs to a device's copy of the kernel: set once per device
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    CFD_CUDA(cudaGetDevice(&dev));
    if (dev > 63 || !(done.load(std::memory_order_relaxed) >> dev & 1ull)) {
        CFD_CUDA(cudaFuncSetAttribute(k_gemm<K, N, EPI>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM));
        if (dev <= 63) done.fetch_or(1ull << dev, std::memory_order_relaxed);
    }
    // the resident blocks of the 152 SMs (each loads the weights once), fewer for few rows
    const unsigned grid = std::min<unsigned>(blocks_for(n, GR * G::WARPS), kTrainChunks * G::PER_SM);
    CFD_LAUNCH_CHAIN((k_gemm<K, N, EPI>), grid, 32 * G::WARPS, G::SMEM, st, n, X1, X2, gate, W,
                     bias, ptr, E, Y, Y2);
    return CFD_OK;
}

int dense_pq(cudaStream_t st, int n, const float* h, const float* W, float* pq) {
    return gemm<HID, 2 * HID, GE_PLAIN>(st, n, h, nullptr, nullptr, W, nullptr, nullptr,
                                              nullptr, pq, nullptr);
}
int dense_update(cudaStream_t st, int n, const float* h, const float* agg, const float* W,
                 const float* b, float* v, float* h1) {
    return gemm<2 * HID, HID, GE_RESIDUAL>(st, n, h, agg, nullptr, W, b, nullptr, nullptr, v,
                                                 h1);
}
int dense_update_bwd(cudaStream_t st, int n, const float* dh, const float* v, const float* W,
                     const int* ptr, float* dhc) {
    return gemm<HID, 2 * HID, GE_SPLIT>(st, n, dh, nullptr, v, W, nullptr, ptr, nullptr,
                                               dhc, nullptr);
}
int dense_pq_bwd(cudaStream_t st, int n, const float* dpq, const float* W, const float* dhc,
                 float* dh) {
    return gemm<2 * HID, HID, GE_ACCUM>(st, n, dpq, nullptr, nullptr, W, nullptr, nullptr,
                                               dhc, dh, nullptr);
}

// h0 = relu(W_in f + b_in); h0 > 0 where the argument is, so it is its own backward mask.  The
// last kEncodeExtra blocks write the layers' dense weights transposed, [input][output] at the same
// offsets of wt, for the forward products (the transposition by each block of each product
// cost 4 to 10 us of 30 to 44).
__global__ void __launch_bounds__(256) k_encode(int n, const float* __restrict__ f,
                                                const float* __restrict__ w,
                                                float* __restrict__ h, float* __restrict__ wt) {
    __shared__ float fs[64 * F_IN];
    w += chain_wait();
    const int tb = (int)blockIdx.x - ((int)gridDim.x - kEncodeExtra);
    if (tb >= 0) {
        for (int q = tb * 256 + threadIdx.x; q < LAYERS * 4 * HID * HID; q += kEncodeExtra * 256) {
            const int off = layer_off(q / (4 * HID * HID)), r = q % (4 * HID * HID);
            if (r < 2 * HID * HID) {
                const int k = r / (2 * HID), c = r % (2 * HID);
                wt[off + L_A + r] = w[off + L_A + c * HID + k];
            } else {
                const int r2 = r - 2 * HID * HID, k = r2 / HID, c = r2 % HID;
                wt[off + L_U + r2] = w[off + L_U + c * 2 * HID + k];
            }
        }
        return;
    }
    const int base = blockIdx.x * 64, o = threadIdx.x & 63;
    for (int q = threadIdx.x; q < 64 * F_IN; q += 256)
        fs[q] = base + q / F_IN < n ? f[(size_t)base * F_IN + q] : 0.f;
    float wr[F_IN];
#pragma unroll
    for (int k = 0; k < F_IN; ++k) wr[k] = w[OFF_W_IN + o * F_IN + k];
    const float b = w[OFF_B_IN + o];
    __syncthreads();
    for (int r = threadIdx.x >> 6; r < 64 && base + r < n; r += 4) {
        float a = b;
#pragma unroll
        for (int k = 0; k < F_IN; ++k) a = fmaf(wr[k], fs[r * F_IN + k], a);
        h[(size_t)(base + r) * HID + o] = fmaxf(a, 0.f);
    }
}

// ------------------------------------------------------------------ weight gradients
// Every weight gradient is a sum over rows, split over kTrainChunks blocks: block c sums its
// rows' contribution to its slice of the parameters into row c of `part` (kTrainChunks x
// (N_PARAMS + 1); the last column is the loss), and k_fold adds the rows in order.
// The fixed chunk count (one block per SM) keeps a step deterministic.
//
// dW[O][I] = sum_r dY[r][O] X[r][I] (and the bias sum_r dY[r][O]) for O x I = 64 x 128 or
// 128 x 64: two groups of 256 threads take alternate rows of a 32-row tile, a thread forms
// 8 x 4 outputs (3 vector loads for 32 FMAs), the next tile's values are loaded while this
// one is summed; with BIAS (O = 64) the columns of dY are summed beside, four rows of a tile a
// thread (by the products' threads they were a fifth of the FP32 operations).  49,794 nodes:
// 128 us + 54 us of fold before (2 shared loads per FMA, 64 rows per partial, 779 partials
// folded by one thread each), 25-32 us now.
template <int O, int I, bool BIAS>
__global__ void __launch_bounds__(512)
k_wgrad(int n, const float* __restrict__ dY, const float* __restrict__ gate,
        const float* __restrict__ X1, const float* __restrict__ X2, float* __restrict__ part,
        int off, int bias_off) {
    constexpr int R = 32, V = R * (O + I) / 4 / 512;  // float4 per thread and tile
    __shared__ __align__(16) float ys[R * O], xs[R * I];
    const int tid = threadIdx.x, grp = tid >> 8, t = tid & 255;
    constexpr int IT = I / 4;
    const int i0 = 4 * (t % IT), o0 = 8 * (t / IT);
    const int rows = (n + kTrainChunks - 1) / kTrainChunks;
    const int b0 = blockIdx.x * rows + chain_wait(), b1 = min(n, b0 + rows);
    static_assert(!BIAS || O == 64, "64 columns by 8 groups of 4 rows");
    const int bo = tid & 63, br = 4 * (tid >> 6);
    float acc[8][4] = {}, bsum = 0.f;
    float4 pre[V];
    auto fetch = [&](int base) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int q = tid + 512 * v;
            float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
            if (q < R * O / 4) {
                const int r = q / (O / 4), c = 4 * (q - r * (O / 4)), row = base + r;
                if (row < b1) {
                    w = *reinterpret_cast<const float4*>(dY + (size_t)row * O + c);
                    if (gate) {
                        const float4 g =
                            *reinterpret_cast<const float4*>(gate + (size_t)row * O + c);
                        w = make_float4(g.x > 0.f ? w.x : 0.f, g.y > 0.f ? w.y : 0.f,
                                        g.z > 0.f ? w.z : 0.f, g.w > 0.f ? w.w : 0.f);
                    }
                }
            } else {
                const int p = q - R * O / 4, r = p / (I / 4), c = 4 * (p - r * (I / 4)),
                          row = base + r;
                if (row < b1)  // one address, not a load on either side of a branch
                    w = *reinterpret_cast<const float4*>((I == 64 || c < 64 ? X1 : X2 - 64) +
                                                         (size_t)row * 64 + c);
            }
            pre[v] = w;
        }
    };
    fetch(b0);
    for (int base = b0; base < b1; base += R) {
        __syncthreads();
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int q = tid + 512 * v;
            if (q < R * O / 4) reinterpret_cast<float4*>(ys)[q] = pre[v];
            else reinterpret_cast<float4*>(xs)[q - R * O / 4] = pre[v];
        }
        __syncthreads();
        if (base + R < b1) fetch(base + R);
        if (BIAS)
#pragma unroll
            for (int u = 0; u < 4; ++u) bsum += ys[(br + u) * O + bo];
#pragma unroll 4
        for (int r = grp; r < R; r += 2) {
            const float4 ya = *reinterpret_cast<const float4*>(ys + r * O + o0);
            const float4 yb = *reinterpret_cast<const float4*>(ys + r * O + o0 + 4);
            const float4 x = *reinterpret_cast<const float4*>(xs + r * I + i0);
            const float y[8] = {ya.x, ya.y, ya.z, ya.w, yb.x, yb.y, yb.z, yb.w};
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                acc[a][0] = fmaf(y[a], x.x, acc[a][0]);
                acc[a][1] = fmaf(y[a], x.y, acc[a][1]);
                acc[a][2] = fmaf(y[a], x.z, acc[a][2]);
                acc[a][3] = fmaf(y[a], x.w, acc[a][3]);
            }
        }
    }
    // group 1 hands its sums to group 0, two output rows at a time (xs holds 256 x 8 floats)
    float* out = part + (size_t)blockIdx.x * (N_PARAMS + 1);
    static_assert(R * I >= 256 * 8, "hand-over buffer");
#pragma unroll
    for (int a = 0; a < 8; a += 2) {
        __syncthreads();
        if (grp == 1) {
            reinterpret_cast<float4*>(xs)[t] = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
            reinterpret_cast<float4*>(xs)[256 + t] =
                make_float4(acc[a + 1][0], acc[a + 1][1], acc[a + 1][2], acc[a + 1][3]);
        }
        __syncthreads();
        if (grp == 0) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float4 q = reinterpret_cast<const float4*>(xs)[256 * u + t];
                // 16-byte aligned: N_PARAMS + 1, the slices' offsets and I are multiples of 4
                *reinterpret_cast<float4*>(out + off + (o0 + a + u) * I + i0) =
                    make_float4(acc[a + u][0] + q.x, acc[a + u][1] + q.y, acc[a + u][2] + q.z,
                                acc[a + u][3] + q.w);
            }
        }
    }
    if (BIAS) {  // ys has been read
        ys[tid] = bsum;
        __syncthreads();
        if (tid < O) {
            float s = 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u) s += ys[64 * u + tid];
            out[bias_off + tid] = s;
        }
    }
}

int wgrad_update(cudaStream_t st, int n, const float* dh, const float* v, const float* h,
                 const float* agg, float* part, int layer) {
    CFD_LAUNCH_CHAIN((k_wgrad<HID, 2 * HID, true>), kTrainChunks, 512, 0, st, n, dh, v, h, agg,
                     part, layer_off(layer) + L_U, layer_off(layer) + L_u);
    return CFD_OK;
}
int wgrad_pq(cudaStream_t st, int n, const float* dpq, const float* h, float* part, int layer) {
    CFD_LAUNCH_CHAIN((k_wgrad<2 * HID, HID, false>), kTrainChunks, 512, 0, st, n, dpq,
                     (const float*)nullptr, h, (const float*)nullptr, part, layer_off(layer) + L_A,
                     -1);
    return CFD_OK;
}

// dW_in, db_in: dh masked by h0 > 0 against the features; thread = output o, rows r mod 8,
// eight rows' loads in flight (78 us with one row at a time at 49,794 nodes, 22 us now)
__global__ void __launch_bounds__(512) k_wgrad_in(int n, const float* __restrict__ dh,
                                                  const float* __restrict__ h0,
                                                  const float* __restrict__ f,
                                                  float* __restrict__ part) {
    constexpr int G = 8, R = 64;
    __shared__ float fs[R * F_IN];
    __shared__ float red[G][64 * (F_IN + 1)];
    const int o = threadIdx.x & 63, g = threadIdx.x >> 6;
    const int rows = (n + kTrainChunks - 1) / kTrainChunks;
    const int b0 = blockIdx.x * rows + chain_wait(), b1 = min(n, b0 + rows);
    float acc[F_IN + 1] = {};
    for (int base = b0; base < b1; base += R) {
        __syncthreads();
        for (int q = threadIdx.x; q < R * F_IN; q += 512)
            fs[q] = base + q / F_IN < b1 ? f[(size_t)base * F_IN + q] : 0.f;
        float d[R / G], m[R / G];
#pragma unroll
        for (int u = 0; u < R / G; ++u) {
            const int r = base + g + G * u;
            d[u] = r < b1 ? dh[(size_t)r * HID + o] : 0.f;
            m[u] = r < b1 ? h0[(size_t)r * HID + o] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < R / G; ++u) {
            const float v = m[u] > 0.f ? d[u] : 0.f;
#pragma unroll
            for (int k = 0; k < F_IN; ++k) acc[k] = fmaf(v, fs[(g + G * u) * F_IN + k], acc[k]);
            acc[F_IN] += v;
        }
    }
#pragma unroll
    for (int k = 0; k <= F_IN; ++k) red[g][k * 64 + o] = acc[k];
    __syncthreads();
    float* out = part + (size_t)blockIdx.x * (N_PARAMS + 1);
    for (int q = threadIdx.x; q < 64 * (F_IN + 1); q += 512) {
        const int k = q >> 6, oo = q & 63;
        float s = 0.f;
#pragma unroll
        for (int u = 0; u < G; ++u) s += red[u][q];
        out[k < F_IN ? OFF_W_IN + oo * F_IN + k : OFF_B_IN + oo] = s;
    }
}

// out[q] = sum over the chunks c, in order, of part[c][q], in four interleaved sums, sixteen
// loads in flight
__global__ void k_fold(int nq, const float* __restrict__ part, float* __restrict__ out,
                       float* __restrict__ loss) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x + chain_wait();
    if (q >= nq) return;
    static_assert(kTrainChunks % 4 == 0, "four sums");
    float a[4] = {};
#pragma unroll 4
    for (int c = 0; c < kTrainChunks; c += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] += part[(size_t)(c + u) * nq + q];
    const float s = (a[0] + a[1]) + (a[2] + a[3]);
    if (q < N_PARAMS) out[q] = s;
    else *loss = s;
}

// ------------------------------------------------------------------ message passing
// 16 lanes per node, four channels each.  Forward: for edge k = (i -> j)
//     z = P_i + Q_j + C e_k + c,   agg_i = sum_k relu(z) / max(deg_i, 1);
// z itself is not kept: the backward pass needs its signs only, 64 bits per edge (bit l of
// plane b: channel 4 l + b), formed by four ballots.  Before, z was written and read back
// per edge and channel (76 MB per layer at 49,794 nodes: 76 + 22 us against 28 us now).  A block
// takes several groups of nodes: C and c are loaded once, and a group's first loads run beside
// the edges of the group before (34 us with a block per 16 nodes).
// A warp takes the nodes i and i + 2 (half_warp_node): structured triangulations alternate
// nodes of 4 and 8 edges, and a warp is as slow as the longer of its two (backward
// 27 us with i and i + 1, 23 so, on such a mesh; on others one pairing is as good as another).
__device__ __forceinline__ int half_warp_node(int half_warp) {
    const int w = half_warp >> 1;
    return 4 * (w >> 1) + (w & 1) + 2 * (half_warp & 1);
}
__global__ void __launch_bounds__(256)
k_edge_fwd(int n, const int* __restrict__ ptr, const int* __restrict__ nbr,
           const float* __restrict__ PQ, const float* __restrict__ e, const float* __restrict__ C,
           const float* __restrict__ c, ushort4* __restrict__ mask, float* __restrict__ agg) {
    const int z = chain_wait();
    const int l = (threadIdx.x & 15) + z, half = threadIdx.x & 16;
    const int at = half_warp_node(threadIdx.x >> 4) + z, nblk = (n + 15) / 16;
    float cw[4][3], cb[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        cb[q] = c[4 * l + q];
#pragma unroll
        for (int u = 0; u < 3; ++u) cw[q][u] = C[(4 * l + q) * 3 + u];
    }
    // a block's 16-node groups; the next group's row pointers and P row load beside this one's edges
    int nk0 = 0, nk1 = 0;
    float4 np = make_float4(0.f, 0.f, 0.f, 0.f);
    auto head = [&](int b) {
        const int i = 16 * b + at;
        if (b >= nblk || i >= n) {
            nk0 = nk1 = 0;
            return;
        }
        nk0 = ptr[i];
        nk1 = ptr[i + 1];
        np = *reinterpret_cast<const float4*>(PQ + (size_t)i * 2 * HID + 4 * l);
    };
    head(blockIdx.x);
    for (int b = blockIdx.x; b < nblk; b += gridDim.x) {
        const int i = 16 * b + at;
        const bool live = i < n;
        const int k0 = nk0, k1 = nk1;
        const float pv[4] = {np.x, np.y, np.z, np.w};
        head(b + gridDim.x);
        float s[4] = {};
        const int deg = k1 - k0, steps = max(deg, __shfl_xor_sync(0xffffffffu, deg, 16));
        constexpr int B = 4;  // edges whose gathers go out together
        for (int t0 = 0; t0 < steps; t0 += B) {
            float4 qv[B];
            float ev[B][3];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int k = k0 + t0 + u;
                qv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                ev[u][0] = ev[u][1] = ev[u][2] = 0.f;
                if (k < k1) {
                    qv[u] = *reinterpret_cast<const float4*>(PQ + (size_t)nbr[k] * 2 * HID + HID + 4 * l);
#pragma unroll
                    for (int q = 0; q < 3; ++q) ev[u][q] = e[3 * (size_t)k + q];
                }
            }
#pragma unroll
            for (int u = 0; u < B; ++u) {
                if (t0 + u >= steps) break;  // the same in the whole warp
                const int k = k0 + t0 + u;
                const float qq[4] = {qv[u].x, qv[u].y, qv[u].z, qv[u].w};
                unsigned short bits[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float z = pv[q] + qq[q] +
                                    (cw[q][0] * ev[u][0] + cw[q][1] * ev[u][1] + cw[q][2] * ev[u][2]) +
                                    cb[q];
                    const bool on = k < k1 && z > 0.f;
                    s[q] += on ? z : 0.f;
                    bits[q] = (unsigned short)(__ballot_sync(0xffffffffu, on) >> half);
                }
                if (l == 0 && k < k1) mask[k] = make_ushort4(bits[0], bits[1], bits[2], bits[3]);
            }
        }
        if (live) {
            const float d = (float)max(deg, 1);
            *reinterpret_cast<float4*>(agg + (size_t)i * HID + 4 * l) =
                make_float4(s[0] / d, s[1] / d, s[2] / d, s[3] / d);
        }
    }
}

// Backward of the messages from g = d agg / deg (the second half of the dhc rows) and the
// signs: with m_k the sign bits of edge k and k' its reverse edge,
//     dP_i = g_i sum_k m_k,   dQ_i = sum_k m_k' g_nbr(k),
//     dC += sum_i g_i sum_k m_k e_k,   dc += sum_i g_i sum_k m_k
// so no per-edge gradient is stored.  kTrainChunks blocks, the nodes interleaved over their
// half-warps; the block's dC, dc go to its row of `part`.  Before: 95 + 53 + 265 + 28 us per
// layer (the edge gradients written, read by the weight gradient and the node sums, the
// partials folded by one block); 23 us now.
__global__ void __launch_bounds__(1024)
k_edge_bwd(int n, const int* __restrict__ ptr, const int* __restrict__ nbr,
           const int* __restrict__ rev, const ushort4* __restrict__ mask,
           const float* __restrict__ dhc, const float* __restrict__ e, float* __restrict__ dPQ,
           float* __restrict__ part, int off) {
    __shared__ float red[16][4 * HID];
    const int z = chain_wait();
    const int l = (threadIdx.x & 15) + z;
    float GC[4][3] = {}, Gc[4] = {};
    const int stride = gridDim.x * 64;
    for (int i = blockIdx.x * 64 + half_warp_node(threadIdx.x >> 4) + z; i < n; i += stride) {
        const int k0 = ptr[i], k1 = ptr[i + 1];
        const float4 g4 = *reinterpret_cast<const float4*>(dhc + (size_t)i * 2 * HID + HID + 4 * l);
        const float g[4] = {g4.x, g4.y, g4.z, g4.w};
        float cnt[4] = {}, S[4][3] = {}, dq[4] = {};
        for (int k = k0; k < k1; ++k) {
            const ushort4 m = mask[k], mr = mask[rev[k]];
            const float4 gj =
                *reinterpret_cast<const float4*>(dhc + (size_t)nbr[k] * 2 * HID + HID + 4 * l);
            const float e0 = e[3 * (size_t)k], e1 = e[3 * (size_t)k + 1], e2 = e[3 * (size_t)k + 2];
            const unsigned short mb[4] = {m.x, m.y, m.z, m.w}, rb[4] = {mr.x, mr.y, mr.z, mr.w};
            const float gv[4] = {gj.x, gj.y, gj.z, gj.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float on = (mb[q] >> l) & 1 ? 1.f : 0.f;
                cnt[q] += on;
                S[q][0] = fmaf(on, e0, S[q][0]);
                S[q][1] = fmaf(on, e1, S[q][1]);
                S[q][2] = fmaf(on, e2, S[q][2]);
                dq[q] += (rb[q] >> l) & 1 ? gv[q] : 0.f;
            }
        }
        float4* o = reinterpret_cast<float4*>(dPQ + (size_t)i * 2 * HID + 4 * l);
        o[0] = make_float4(g[0] * cnt[0], g[1] * cnt[1], g[2] * cnt[2], g[3] * cnt[3]);
        o[HID / 4] = make_float4(dq[0], dq[1], dq[2], dq[3]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int u = 0; u < 3; ++u) GC[q][u] = fmaf(g[q], S[q][u], GC[q][u]);
            Gc[q] = fmaf(g[q], cnt[q], Gc[q]);
        }
    }
    // fold the block's 64 half-warps: the two of a warp by a shuffle, then 16 rows of shared
    // memory twice, then the rows in order
    float v[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int u = 0; u < 3; ++u) v[3 * q + u] = GC[q][u];
        v[12 + q] = Gc[q];
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], 16);
    const int w = threadIdx.x >> 5;
    for (int pass = 0; pass < 2; ++pass) {
        if ((w >> 4) == pass && (threadIdx.x & 31) < 16)
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                float& d = red[w & 15][q < 12 ? (4 * l + q / 3) * 3 + q % 3 : 3 * HID + 4 * l + (q - 12)];
                d = pass ? d + v[q] : v[q];
            }
        __syncthreads();
    }
    if (threadIdx.x < 4 * HID) {
        float s = 0.f;
#pragma unroll
        for (int r = 0; r < 16; ++r) s += red[r][threadIdx.x];
        part[(size_t)blockIdx.x * (N_PARAMS + 1) + off + threadIdx.x] = s;  // C (64 x 3), then c
    }
}

// ------------------------------------------------------------------ decoder, loss and Adam
// y = W_out h + b_out, four lanes per node with 16 channels each.  With a target also the
// loss |y - t|^2 over the free nodes, dy = 2 (y - t) / nfree, dh = W_out^T dy, and the
// block's share of dW_out, db_out and the loss in its row of `part`.
__global__ void __launch_bounds__(256)
k_decode(int n, const float* __restrict__ h, const float* __restrict__ w, float* __restrict__ y,
         const float* __restrict__ target, const int* __restrict__ kind, float inv_nfree,
         float* __restrict__ dh, float* __restrict__ part) {
    __shared__ float red[8][(HID + 1) * OUT + 1];
    const int z = chain_wait(), l = (threadIdx.x & 3) + z;
    float wo[OUT][16], GW[OUT][16] = {}, gb[OUT] = {}, loss = 0.f;
#pragma unroll
    for (int o = 0; o < OUT; ++o)
#pragma unroll
        for (int k = 0; k < 16; ++k) wo[o][k] = w[OFF_W_OUT + o * HID + 16 * l + k];
    const int stride = gridDim.x * 64;
    // whole warps walk the loop together (the shuffles below)
    for (int i0 = blockIdx.x * 64 + 8 * (threadIdx.x >> 5) + z; i0 < n; i0 += stride) {
        const int i = i0 + ((threadIdx.x & 31) >> 2);
        float hv[16];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < n) q = *reinterpret_cast<const float4*>(h + (size_t)i * HID + 16 * l + 4 * v);
            hv[4 * v] = q.x;
            hv[4 * v + 1] = q.y;
            hv[4 * v + 2] = q.z;
            hv[4 * v + 3] = q.w;
        }
        float d[OUT];
#pragma unroll
        for (int o = 0; o < OUT; ++o) {
            float a = l == 0 ? w[OFF_B_OUT + o] : 0.f;
#pragma unroll
            for (int k = 0; k < 16; ++k) a = fmaf(wo[o][k], hv[k], a);
            a += __shfl_xor_sync(0xffffffffu, a, 1);
            a += __shfl_xor_sync(0xffffffffu, a, 2);
            if (l == 0 && i < n) y[(size_t)OUT * i + o] = a;
            d[o] = a;
        }
        if (!target || i >= n) continue;
        const bool fr = kind[i] == KIND_FREE;
        float4 g[4];
        float* gf = reinterpret_cast<float*>(g);
#pragma unroll
        for (int k = 0; k < 16; ++k) gf[k] = 0.f;
#pragma unroll
        for (int o = 0; o < OUT; ++o) {
            const float df = fr ? d[o] - target[(size_t)OUT * i + o] : 0.f;
            const float dy = 2.f * df * inv_nfree;
            if (l == 0) {
                loss += df * df;
                gb[o] += dy;
            }
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                gf[k] = fmaf(dy, wo[o][k], gf[k]);
                GW[o][k] = fmaf(dy, hv[k], GW[o][k]);
            }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v)
            *reinterpret_cast<float4*>(dh + (size_t)i * HID + 16 * l + 4 * v) = g[v];
    }
    if (!target) return;
    // the eight nodes of a warp, then the eight warps in order
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto fold = [&](float v, int at) {
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (lane < 4 && at >= 0) red[wp][at] = v;
    };
#pragma unroll
    for (int o = 0; o < OUT; ++o) {
#pragma unroll
        for (int k = 0; k < 16; ++k) fold(GW[o][k], o * HID + 16 * l + k);
        fold(gb[o], l == 0 ? OUT * HID + o : -1);
    }
    fold(loss, l == 0 ? OUT * HID + OUT : -1);
    __syncthreads();
    for (int q = threadIdx.x; q < (HID + 1) * OUT + 1; q += 256) {
        float s = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) s += red[r][q];
        part[(size_t)blockIdx.x * (N_PARAMS + 1) + OFF_W_OUT + q] = s;  // b_out, the loss follow
    }
}

__global__ void k_adam(int np, float* __restrict__ w, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2,
                       float eps, float bc1, float bc2) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= np) return;
    const float gq = g[q];
    const float mq = b1 * m[q] + (1.f - b1) * gq;
    const float vq = b2 * v[q] + (1.f - b2) * gq * gq;
    m[q] = mq;
    v[q] = vq;
    const float mh = mq / bc1, vh = vq / bc2;
    w[q] = w[q] - lr * mh / (sqrtf(vh) + eps);
}

// training targets: the fields (Phi, Psi_x, Psi_y) of the plain solve, stored as
// (Phi, Psi_x / L, Psi_y / L)
__global__ void k_targets(int n, const double* __restrict__ phi, const double* __restrict__ psx,
                          const double* __restrict__ psy, const Globals* __restrict__ G,
                          float* __restrict__ t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double iL = 1.0 / G->L;
    t[OUT * i] = (float)phi[i];
    t[OUT * i + 1] = (float)(psx[i] * iL);
    t[OUT * i + 2] = (float)(psy[i] * iL);
}

// guess at free nodes: u = t Phi + L M (Psi_x/L, Psi_y/L); boundary nodes keep their
// prescribed values
__global__ void k_guess(int n, const float* __restrict__ y, const int* __restrict__ kind,
                        const double* __restrict__ gnx, const double* __restrict__ gny,
                        const Globals* __restrict__ G, double* __restrict__ ux,
                        double* __restrict__ uy, const int* __restrict__ gate) {
    if (gate && !*gate) return;
    const Globals g = *G;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (kind[i] != KIND_FREE) {
            ux[i] = gnx[i];
            uy[i] = gny[i];
            continue;
        }
        const double phi = y[OUT * i], px = g.L * (double)y[OUT * i + 1],
                     py = g.L * (double)y[OUT * i + 2];
        ux[i] = g.tx * phi + g.m11 * px + g.m12 * py;
        uy[i] = g.ty * phi + g.m21 * px + g.m22 * py;
    }
}

}  // namespace mpnn
}  // namespace cfd

namespace cfd {
namespace mpnn {

// ------------------------------------------------------------------ BF16 inference
// Tensor-core pass (mma.sync m16n8k16, BF16 operands, FP32 accumulation).  A warp owns 16
// nodes, a block of IW warps a tile of 16*IW nodes; blocks loop over tiles so that each
// loads the layer's weights into shared memory once.  Per layer one kernel: the message
// aggregation of the layer (FP32 arithmetic on the BF16 P, Q of the previous kernel), the
// update GEMM U [h; agg], the residual, then the next layer's P|Q GEMM or, after the last
// layer, the decoder.  P|Q alternates between two buffers.
constexpr int IW = 8;
constexpr int TILE = 16 * IW;
constexpr int XS = 2 * HID + 8;  // shared row stride (bf16) of 128-wide tiles
constexpr int HS = HID + 8;      // of 64-wide tiles (the +8 keeps fragment loads
                                 // free of bank conflicts)
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ unsigned ld_b32(const bf16* p) {
    return *reinterpret_cast<const unsigned*>(p);
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2,
                                         unsigned a3, unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// acc[nt] += X[16][K] . W[nt*8 .. nt*8+8)[K]^T, X and W in shared memory (row strides xs,
// ws in elements).  Fragment layout of m16n8k16: lane = 4 g + t; A rows g and g+8, columns
// 2t, 2t+1 (+8); B column g, rows 2t, 2t+1 (+8); D rows g and g+8, columns 2t, 2t+1.
template <int K, int NT>
__device__ __forceinline__ void warp_gemm(const bf16* X, int xs, const bf16* W, int ws,
                                          float (&acc)[NT][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int kk = 0; kk < K / 16; ++kk) {
        const int k0 = kk * 16 + 2 * t;
        const unsigned a0 = ld_b32(X + g * xs + k0);
        const unsigned a1 = ld_b32(X + (g + 8) * xs + k0);
        const unsigned a2 = ld_b32(X + g * xs + k0 + 8);
        const unsigned a3 = ld_b32(X + (g + 8) * xs + k0 + 8);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const bf16* wr = W + (nt * 8 + g) * ws + k0;
            mma_bf16(acc[nt], a0, a1, a2, a3, ld_b32(wr), ld_b32(wr + 8));
        }
    }
}

// D (16 x NT*8, FP32 fragments) -> global rows base.. (row stride ld), BF16
template <int NT>
__device__ __forceinline__ void store_tile_bf16(const float (&acc)[NT][4], int base, int n, bf16* out,
                                                int ld) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int col = nt * 8 + 2 * t;
        if (base + g < n)
            *reinterpret_cast<__nv_bfloat162*>(out + (size_t)(base + g) * ld + col) =
                __floats2bfloat162_rn(acc[nt][0], acc[nt][1]);
        if (base + g + 8 < n)
            *reinterpret_cast<__nv_bfloat162*>(out + (size_t)(base + g + 8) * ld + col) =
                __floats2bfloat162_rn(acc[nt][2], acc[nt][3]);
    }
}

__global__ void k_to_bf16(int np, const float* __restrict__ w, bf16* __restrict__ wb) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < np) wb[q] = __float2bfloat16_rn(w[q]);
}

// rows x cols of a row-major BF16 matrix into shared memory with row stride ld
__device__ __forceinline__ void load_mat(bf16* dst, int ld, const bf16* src, int rows, int cols) {
    for (int q = threadIdx.x; q < rows * cols / 2; q += blockDim.x) {
        const int r = (2 * q) / cols, c = 2 * q - r * cols;
        *reinterpret_cast<unsigned*>(dst + r * ld + c) =
            *reinterpret_cast<const unsigned*>(src + (size_t)r * cols + c);
    }
}

// h0 = relu(W_in f + b_in) (FP32), then P|Q of layer 0
__global__ void __launch_bounds__(32 * IW) k_infer_encode(int n, const float* __restrict__ f,
                                                          const float* __restrict__ w,
                                                          const bf16* __restrict__ wb,
                                                          bf16* __restrict__ hb,
                                                          bf16* __restrict__ pq_out,
                                                          const int* __restrict__ gate) {
    if (gate && !*gate) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* Ws = reinterpret_cast<bf16*>(smem_raw);   // 128 x HS: [A0; B0]
    bf16* Hs = Ws + 2 * HID * HS;                    // IW x 16 x HS
    float* Wi = reinterpret_cast<float*>(Hs + IW * 16 * HS);  // HID x F_IN, then b_in
    load_mat(Ws, HS, wb + layer_off(0) + L_A, 2 * HID, HID);
    for (int q = threadIdx.x; q < HID * F_IN + HID; q += blockDim.x) Wi[q] = w[OFF_W_IN + q];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bf16* H = Hs + warp * 16 * HS;
    const int ntile = (n + TILE - 1) / TILE;
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int base = tile * TILE + warp * 16;
        {  // all 16 nodes at once: lane l owns node l/2 and the outputs [32 (l%2), +32)
            const int r = lane >> 1, o0 = 32 * (lane & 1), node = base + r;
            float fi[F_IN];
#pragma unroll
            for (int k = 0; k < F_IN; ++k) fi[k] = node < n ? f[(size_t)node * F_IN + k] : 0.f;
            unsigned w16[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                float hv[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int o = o0 + 2 * q + u;
                    float a = Wi[HID * F_IN + o];
#pragma unroll
                    for (int k = 0; k < F_IN; ++k) a += Wi[o * F_IN + k] * fi[k];
                    hv[u] = node < n ? fmaxf(a, 0.f) : 0.f;
                }
                const __nv_bfloat162 h2 = __floats2bfloat162_rn(hv[0], hv[1]);
                w16[q] = *reinterpret_cast<const unsigned*>(&h2);
            }
            uint4* hs = reinterpret_cast<uint4*>(H + r * HS + o0);
            uint4* hg = reinterpret_cast<uint4*>(hb + (size_t)node * HID + o0);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const uint4 w = make_uint4(w16[4 * v], w16[4 * v + 1], w16[4 * v + 2], w16[4 * v + 3]);
                hs[v] = w;
                if (node < n) hg[v] = w;
            }
        }
        __syncwarp();
        float acc[16][4];
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        warp_gemm<HID, 16>(H, HS, Ws, HS, acc);
        store_tile_bf16<16>(acc, base, n, pq_out, 2 * HID);
        __syncwarp();
    }
}

// layer l: aggregation, update GEMM, residual; then P|Q of layer l+1 (wb_next) or the
// decoder (wb_next == null)
__global__ void __launch_bounds__(32 * IW, 2) k_infer_layer(
    int n, int l, const int* __restrict__ ptr, const int* __restrict__ nbr,
    const float* __restrict__ e, const float* __restrict__ w, const bf16* __restrict__ wb,
    int has_next, const bf16* __restrict__ pq_in, bf16* __restrict__ hb,
    bf16* __restrict__ pq_out, float* __restrict__ y, const int* __restrict__ gate) {
    if (gate && !*gate) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* Us = reinterpret_cast<bf16*>(smem_raw);  // HID x XS
    bf16* Ws = Us + HID * XS;                       // 128 x HS: [A; B] of layer l+1
    bf16* Xs = Ws + 2 * HID * HS;                   // IW x 16 x XS
    float* Cs = reinterpret_cast<float*>(Xs + IW * 16 * XS);  // C (HID x 3), c, u
    float* cs = Cs + HID * E_F;
    float* us = cs + HID;
    const float* W = w + layer_off(l);
    load_mat(Us, XS, wb + layer_off(l) + L_U, HID, 2 * HID);
    if (has_next) load_mat(Ws, HS, wb + layer_off(l + 1) + L_A, 2 * HID, HID);
    for (int q = threadIdx.x; q < HID * E_F; q += blockDim.x) Cs[q] = W[L_C + q];
    for (int q = threadIdx.x; q < HID; q += blockDim.x) {
        cs[q] = W[L_c + q];
        us[q] = W[L_u + q];
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    bf16* X = Xs + warp * 16 * XS;
    const int o0 = 2 * lane;
    const int ntile = (n + TILE - 1) / TILE;
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int base = tile * TILE + warp * 16;
        // [h; agg] rows of the warp's 16 nodes, 8 at a time: lane l owns node l/4 (+8) and
        // the 16 features [16 (l%4), 16 (l%4) + 16); rows are read as 16-byte vectors
        for (int pass = 0; pass < 2; ++pass) {
            const int r = (lane >> 2) + 8 * pass, f0 = 16 * (lane & 3), node = base + r;
            float acc16[16], pz[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) acc16[q] = 0.f;
            uint4 hv4[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
            if (node < n) {
                const uint4* hp = reinterpret_cast<const uint4*>(hb + (size_t)node * HID + f0);
                const uint4* pp = reinterpret_cast<const uint4*>(pq_in + (size_t)node * 2 * HID + f0);
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    hv4[v] = hp[v];
                    const uint4 pv = pp[v];
                    const unsigned w4[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float2 f2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w4[u]));
                        pz[8 * v + 2 * u] = f2.x + cs[f0 + 8 * v + 2 * u];  // P_i + c
                        pz[8 * v + 2 * u + 1] = f2.y + cs[f0 + 8 * v + 2 * u + 1];
                    }
                }
                const int k0 = ptr[node], k1 = ptr[node + 1];
                for (int k = k0; k < k1; ++k) {
                    const int j = nbr[k];
                    const float e0 = e[3 * (size_t)k], e1 = e[3 * (size_t)k + 1],
                                e2 = e[3 * (size_t)k + 2];
                    const uint4* qp =
                        reinterpret_cast<const uint4*>(pq_in + (size_t)j * 2 * HID + HID + f0);
                    const uint4 qa = qp[0], qb = qp[1];
                    const unsigned w8[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const float2 q2 =
                            __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w8[u]));
                        const int o = f0 + 2 * u;
                        const float z0 = pz[2 * u] + q2.x +
                                         (Cs[o * 3] * e0 + Cs[o * 3 + 1] * e1 + Cs[o * 3 + 2] * e2);
                        const float z1 = pz[2 * u + 1] + q2.y +
                                         (Cs[o * 3 + 3] * e0 + Cs[o * 3 + 4] * e1 + Cs[o * 3 + 5] * e2);
                        acc16[2 * u] += fmaxf(z0, 0.f);
                        acc16[2 * u + 1] += fmaxf(z1, 0.f);
                    }
                }
                const float inv = 1.f / (float)max(k1 - k0, 1);
#pragma unroll
                for (int q = 0; q < 16; ++q) acc16[q] *= inv;
            }
            uint4* xh = reinterpret_cast<uint4*>(X + r * XS + f0);
            uint4* xa = reinterpret_cast<uint4*>(X + r * XS + HID + f0);
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                xh[v] = hv4[v];
                unsigned w4[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const __nv_bfloat162 b2 =
                        __floats2bfloat162_rn(acc16[8 * v + 2 * u], acc16[8 * v + 2 * u + 1]);
                    w4[u] = *reinterpret_cast<const unsigned*>(&b2);
                }
                xa[v] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
        }
        __syncwarp();
        float acc[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        warp_gemm<2 * HID, 8>(X, XS, Us, XS, acc);
        __syncwarp();
        // h <- h + relu(v + u), written back over the h half of the tile and to hb
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int col = nt * 8 + 2 * t;
#pragma unroll
            for (int hlf = 0; hlf < 2; ++hlf) {
                const int row = g + 8 * hlf;
                const float2 hv = __bfloat1622float2(
                    *reinterpret_cast<const __nv_bfloat162*>(X + row * XS + col));
                const float n0 = hv.x + fmaxf(acc[nt][2 * hlf] + us[col], 0.f);
                const float n1 = hv.y + fmaxf(acc[nt][2 * hlf + 1] + us[col + 1], 0.f);
                const __nv_bfloat162 nh = __floats2bfloat162_rn(n0, n1);
                *reinterpret_cast<__nv_bfloat162*>(X + row * XS + col) = nh;
                if (base + row < n)
                    *reinterpret_cast<__nv_bfloat162*>(hb + (size_t)(base + row) * HID + col) = nh;
            }
        }
        __syncwarp();
        if (has_next) {
            float acc2[16][4];
#pragma unroll
            for (int nt = 0; nt < 16; ++nt)
                acc2[nt][0] = acc2[nt][1] = acc2[nt][2] = acc2[nt][3] = 0.f;
            warp_gemm<HID, 16>(X, XS, Ws, HS, acc2);
            store_tile_bf16<16>(acc2, base, n, pq_out, 2 * HID);
        } else {
            // decoder: 16 nodes x OUT outputs over the warp's lanes
            for (int q = lane; q < 16 * OUT; q += 32) {
                const int r = q / OUT, o = q - r * OUT, node = base + r;
                float a = w[OFF_B_OUT + o];
                for (int k = 0; k < HID; ++k)
                    a += w[OFF_W_OUT + o * HID + k] * __bfloat162float(X[r * XS + k]);
                if (node < n) y[(size_t)OUT * node + o] = a;
            }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ BF16 inference, tcgen05
// The same passes with the GEMMs on the 5th-generation tensor cores.  A block of 8 warps
// owns a tile of 128 nodes (the MMA's M): the warps gather the tile's [h; agg] rows (16
// nodes each, the arithmetic of the mma.sync pass) into shared memory, one thread issues
// tcgen05.mma (BF16 operands from shared memory, FP32 accumulators in tensor memory) and
// commits it to an mbarrier, and after the bounded wait every warp reads its 32 rows of
// the accumulator with tcgen05.ld for the epilogue.  The update GEMM (N = 64, K = 128) and
// the next layer's P|Q GEMM (N = 128, K = 64) use the same 128 tensor-memory columns one
// after the other.
//
// The gather bounds a layer, by the latency of its loads (row pointer, neighbour, neighbour's
// Q row) as long as few of them are in flight.  So the tile's neighbours and edge features,
// contiguous in both arrays, come by cp.async.bulk while the block finishes the tile before;
// eight lanes take a node (eight channels each, C's 24 coefficients in registers) and have
// the Q rows of up to eight edges in flight; and every global row goes out through shared
// memory, so that a warp writes whole lines.  1,048,576 nodes, 6.3 M edges: 480 us a layer
// with one edge in flight per lane and rows stored by their owner threads, 312 us now; the
// encoder pass 194 us, 118 us now.
namespace tc {
constexpr int TM = 128;          // nodes per tile
constexpr int NTHR = 256;        // 8 warps
constexpr unsigned TMEM_COLS = 128;
// K-major operands in the no-swizzle core-matrix layout: a core matrix is 8 rows x 16
// bytes (128 contiguous bytes); the core matrices of one 8-row group lie along K, 128 B
// apart (the descriptor's leading byte offset); the 8-row groups lie SBO bytes apart.
// The tile's core matrices lie 144 B apart: lanes that write one row's chunks hit different banks.
constexpr int LBO = 128;
constexpr int LBO_X = 144;
constexpr int SBO_X = LBO_X * 2 * HID / 8;  // the tile, 128 rows x K = 128 (h, then agg)
constexpr int SBO_U = 16 * 2 * HID;  // U: N = 64 rows x K = 128
constexpr int SBO_W = 16 * HID;      // [A; B]: N = 128 rows x K = 64
constexpr int X_BYTES = TM / 8 * SBO_X;
constexpr int PQ_ROW = 2 * 2 * HID + 16;  // a staged P|Q row (padded: rows in different banks)
constexpr int PQ_BLK = X_BYTES / 4;       // 32 of them: the rows of one quarter of the tile
static_assert(32 * PQ_ROW <= PQ_BLK, "staged P|Q rows");
constexpr int GB = 3;                     // edges of a batch
constexpr int EC = 1024;                  // staged edges (a tile of more reads global memory)
constexpr int U_BYTES = HID * 2 * HID * 2;
constexpr int W_BYTES = 2 * HID * HID * 2;
constexpr int F_FLOATS = HID * F_IN + HID;  // the largest float table (W_in, b_in)
static_assert(HID * E_F + 2 * HID + OUT * HID + OUT <= F_FLOATS, "float tables");
static_assert(F_FLOATS % 4 == 0 && EC % 4 == 0, "16-byte offsets");
constexpr int SMEM = X_BYTES + U_BYTES + W_BYTES + 4 * F_FLOATS + 16 * EC + 32;

__host__ __device__ constexpr int cm_off(int r, int k, int sbo, int lbo = LBO) {
    return (r >> 3) * sbo + (k >> 3) * lbo + (r & 7) * 16 + (k & 7) * 2;
}
__host__ __device__ constexpr int x_off(int r, int k) { return cm_off(r, k, SBO_X, LBO_X); }

// shared-memory matrix descriptor: start address, leading and stride byte offsets (all
// >> 4), the descriptor version 1 at bit 46, base offset 0, no swizzle
__device__ __forceinline__ unsigned long long sdesc(unsigned saddr, unsigned sbo, unsigned lbo) {
    return (unsigned long long)((saddr & 0x3FFFFu) >> 4) |
           ((unsigned long long)(lbo >> 4) << 16) | ((unsigned long long)(sbo >> 4) << 32) |
           (1ull << 46);
}

// instruction descriptor of kind::f16: FP32 accumulator (bit 4), A and B BF16 (bits 7,
// 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr unsigned idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) |
           ((unsigned)(m >> 4) << 24);
}

__device__ __forceinline__ unsigned su32(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// this thread's st.shared become visible to the tensor cores' reads
__device__ __forceinline__ void fence_smem_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mma(unsigned d, unsigned long long a, unsigned long long b,
                                    unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        :
        : "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void commit(unsigned mbar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
        : "memory");
}

// bounded wait on the mbarrier's phase of the given parity (mbar_wait_bounded)
__device__ __forceinline__ bool wait_parity(unsigned mbar, unsigned parity) {
    return mbar_wait_bounded(mbar, parity);
}

// 16 consecutive FP32 columns of this thread's tensor-memory lane; the wait is tied to
// the registers so that no use moves above it
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float (&v)[16]) {
    unsigned r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// rows x cols of a row-major BF16 matrix into the core-matrix layout (16-byte chunks)
__device__ __forceinline__ void load_cm(unsigned char* dst, int sbo, const bf16* src, int rows,
                                        int cols) {
    const int per_row = cols / 8;
    for (int q = threadIdx.x; q < rows * per_row; q += blockDim.x) {
        const int r = q / per_row, k = (q - r * per_row) * 8;
        *reinterpret_cast<uint4*>(dst + cm_off(r, k, sbo)) =
            *reinterpret_cast<const uint4*>(src + (size_t)r * cols + k);
    }
}

__device__ __forceinline__ unsigned pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned*>(&h);
}

__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_copy(unsigned dst, const void* src, unsigned bytes, unsigned mbar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(dst), "l"(src), "r"(bytes), "r"(mbar)
        : "memory");
}
// the two warps that share a quarter of the tile
__device__ __forceinline__ void pair_sync(int q4) {
    asm volatile("bar.sync %0, 64;" ::"r"(1 + q4) : "memory");
}
__device__ __forceinline__ void unpack8(const uint4 v, float (&x)[8]) {
    const unsigned w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const float2 f2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w4[u]));
        x[2 * u] = f2.x;
        x[2 * u + 1] = f2.y;
    }
}
// two FP32 operations in one instruction, each rounded as the single one
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpair(f32x2 p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// a BF16 pair as two floats
__device__ __forceinline__ f32x2 widen2(unsigned v) {
    return pair(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
    return make_uint4(pack2(x[0], x[1]), pack2(x[2], x[3]), pack2(x[4], x[5]), pack2(x[6], x[7]));
}

// ENC: h0 = relu(W_in f + b_in), then P|Q of layer 0.  Otherwise layer l: aggregation,
// update GEMM, residual, then P|Q of layer l+1 (has_next) or the decoder.  nbr and e are
// readable up to the next 16-byte boundary.
template <bool ENC>
__global__ void __launch_bounds__(NTHR, 2) k_infer_tc(
    int n, int l, const int* __restrict__ ptr, const int* __restrict__ nbr,
    const float* __restrict__ e, const float* __restrict__ f, const float* __restrict__ w,
    const bf16* __restrict__ wb, int has_next, const bf16* __restrict__ pq_in,
    bf16* __restrict__ hb, bf16* __restrict__ pq_out, float* __restrict__ y,
    const int* __restrict__ gate, int* __restrict__ err) {
    if (gate && !*gate) {
        chain_wait();
        return;
    }
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* Xs = smem_raw;
    unsigned char* Us = Xs + X_BYTES;
    unsigned char* Ws = Us + U_BYTES;
    float* fl = reinterpret_cast<float*>(Ws + W_BYTES);
    int* sn = reinterpret_cast<int*>(fl + F_FLOATS);       // the tile's neighbours ..
    float* se = reinterpret_cast<float*>(sn + EC);          // .. and edge features
    unsigned long long* mbar = reinterpret_cast<unsigned long long*>(se + 3 * EC);
    unsigned* tslot = reinterpret_cast<unsigned*>(mbar + 2);
    int* abort_flag = reinterpret_cast<int*>(tslot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // float tables: ENC W_in (transposed), b_in; layers C, c, u, W_out, b_out
    float *Cs = fl, *cs = fl + HID * E_F, *us = cs + HID, *wo = us + HID;
    const int has_pq = ENC || has_next;
    if (ENC) {
        for (int q = tid; q < HID * F_IN; q += NTHR)
            fl[(q % F_IN) * HID + q / F_IN] = w[OFF_W_IN + q];
        for (int q = tid; q < HID; q += NTHR) fl[HID * F_IN + q] = w[OFF_W_IN + HID * F_IN + q];
    } else {
        const float* W = w + layer_off(l);
        load_cm(Us, SBO_U, wb + layer_off(l) + L_U, HID, 2 * HID);
        for (int q = tid; q < HID * E_F; q += NTHR) Cs[q] = W[L_C + q];
        for (int q = tid; q < HID; q += NTHR) {
            cs[q] = W[L_c + q];
            us[q] = W[L_u + q];
        }
        if (!has_next)
            for (int q = tid; q < OUT * HID + OUT; q += NTHR) wo[q] = w[OFF_W_OUT + q];
    }
    if (has_pq) load_cm(Ws, SBO_W, wb + layer_off(ENC ? 0 : l + 1) + L_A, 2 * HID, HID);
    const unsigned ubar = su32(mbar), sbar = su32(mbar + 1);  // the MMAs, the staged edges
    if (tid == 0) {
        *abort_flag = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ubar) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         su32(tslot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_smem_async();
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tbase = *tslot;
    const unsigned xa = su32(Xs), ua = su32(Us), wa = su32(Ws);
    // epilogue geometry: warp w reads tensor-memory lanes 32 (w % 4) .. (its 32 rows) and
    // half w / 4 of the accumulator's columns; it writes the rows 16 (w / 4) .. of them out
    const int q4 = warp & 3, half = warp >> 2;
    const int erow = 32 * q4 + lane;
    const unsigned tlane = tbase + ((unsigned)(32 * q4) << 16);
    // gather geometry: lane l takes node l / 8 of the pass and the channels 8 (l % 8) ..
    const int sub = lane >> 3, f0 = 8 * (lane & 7);
    unsigned phase = 0, sphase = 0;
    bool pending = false;   // a commit that this block has not seen arrive
    bool spending = false;  // staged edges that this thread has not seen arrive
    f32x2 C0[4], C1[4], C2[4];
    if (!ENC)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* c = Cs + 3 * (f0 + 2 * i);
            C0[i] = pair(c[0], c[3]);
            C1[i] = pair(c[1], c[4]);
            C2[i] = pair(c[2], c[5]);
        }
    const int ntile = (n + TM - 1) / TM;
    // the row pointers of a tile: its first and last edge, and this warp's nodes (lanes 0..16)
    int tk0 = 0, tk1 = 0, pv = 0;
    auto pointers = [&](int tile, int& k0, int& k1, int& v) {
        const int tb = tile * TM;
        k0 = ptr[tb];
        k1 = ptr[min(tb + TM, n)];
        v = ptr[min(tb + 16 * warp + min(lane, 16), n)];
    };
    // edges [tk0, tk1) into shared memory, from the 16-byte boundary before the first
    auto stage = [&]() {
        const int ka = tk0 & ~3, cnt = tk1 - ka;
        spending = tk1 > tk0 && cnt <= EC;
        if (spending && tid == NTHR - 32) {
            const unsigned nbytes = (4u * cnt + 15u) & ~15u, ebytes = (12u * cnt + 15u) & ~15u;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sbar),
                         "r"(nbytes + ebytes)
                         : "memory");
            bulk_copy(su32(sn), nbr + ka, nbytes, sbar);
            bulk_copy(su32(se), e + 3 * (size_t)ka, ebytes, sbar);
        }
    };
    if (!ENC && (int)blockIdx.x < ntile) {
        pointers(blockIdx.x, tk0, tk1, pv);
        stage();
    }
    // What is above reads only what no kernel of the pass writes (weights, rows, edges): a block
    // sets itself up while the layer ahead drains.  1,048,576 nodes: 1.542 -> 1.524 ms a pass; a
    // smaller mesh 0.887 -> 0.869.
    const int z = chain_wait();
    hb += z;
    pq_in += z;
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int tb = tile * TM;
        const bool more = tile + (int)gridDim.x < ntile;
        int nk0 = 0, nk1 = 0, nv = 0;
        if (!ENC && more) pointers(tile + gridDim.x, nk0, nk1, nv);
        if (ENC) {
            // lane l of warp w owns row 16 w + l / 2 and every other chunk of eight outputs
            const int r = 16 * warp + (lane >> 1), node = tb + r;
            float fi[F_IN];
            static_assert(F_IN % 2 == 0, "float2 rows");
#pragma unroll
            for (int k = 0; k < F_IN; k += 2) {
                const float2 v = node < n ? *reinterpret_cast<const float2*>(f + (size_t)node * F_IN + k)
                                          : make_float2(0.f, 0.f);
                fi[k] = v.x;
                fi[k + 1] = v.y;
            }
#pragma unroll
            for (int v = 0; v < HID / 16; ++v) {
                const int o = 16 * v + 8 * (lane & 1);
                float a[8];
#pragma unroll
                for (int k = -1; k < F_IN; ++k) {
                    const float4* wk =
                        reinterpret_cast<const float4*>(fl + (k < 0 ? HID * F_IN : k * HID) + o);
                    const float4 wl = wk[0], wh = wk[1];
                    const float wv[8] = {wl.x, wl.y, wl.z, wl.w, wh.x, wh.y, wh.z, wh.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (k < 0) a[i] = wv[i];
                        else a[i] += wv[i] * fi[k < 0 ? 0 : k];
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) a[i] = node < n ? fmaxf(a[i], 0.f) : 0.f;
                *reinterpret_cast<uint4*>(Xs + x_off(r, o)) = pack8(a);
            }
        } else {
            // [h; agg] rows: eight lanes take four nodes, one after the other
            const int r0 = 16 * warp + 4 * sub, nb0 = tb + r0, ka = tk0 & ~3;
            const bool staged = spending;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool in = nb0 + i < n;
                cp_async16(xa + x_off(r0 + i, f0), hb + (in ? (size_t)(nb0 + i) * HID + f0 : 0),
                           in ? 16 : 0);
            }
            const uint4* prow = reinterpret_cast<const uint4*>(pq_in + f0);
            const uint4* qrow = reinterpret_cast<const uint4*>(pq_in + HID + f0);
            uint4 pnext = nb0 < n ? prow[(size_t)nb0 * (2 * HID / 8)] : make_uint4(0u, 0u, 0u, 0u);
            bool here = true;  // nothing is gathered by indices that did not arrive
            if (staged) {
                here = __all_sync(0xffffffffu, wait_parity(sbar, sphase & 1));
                if (here) {
                    spending = false;
                    sphase += 1;
                } else {
                    atomicExch(err, (int)CFD_ERR_BARRIER);
                    *abort_flag = 1;
                }
            }
            auto gather = [&](auto from_stage) {
                constexpr bool STAGED = decltype(from_stage)::value;
                int ke[5];  // the four nodes' first edges and the end of the last
#pragma unroll
                for (int i = 0; i < 5; ++i) ke[i] = __shfl_sync(0xffffffffu, pv, 4 * sub + i);
                const int kn = ke[4];
                int i = 0, k1 = ke[1], deg = ke[1] - ke[0];
                f32x2 pz[4], acc[4];
                auto open = [&]() {  // node i: z's part that its edges share, an empty sum
                    const unsigned pw[4] = {pnext.x, pnext.y, pnext.z, pnext.w};
                    if (i < 3 && nb0 + i + 1 < n) pnext = prow[(size_t)(nb0 + i + 1) * (2 * HID / 8)];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        pz[c] = add2(widen2(pw[c]), pair(cs[f0 + 2 * c], cs[f0 + 2 * c + 1]));
                        acc[c] = 0ull;
                    }
                };
                auto close = [&]() {  // the mean message of node i; on to the next
                    const float inv = 1.f / (float)max(deg, 1);
                    unsigned aw[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float2 m = unpair(acc[c]);
                        aw[c] = pack2(m.x * inv, m.y * inv);
                    }
                    *reinterpret_cast<uint4*>(Xs + x_off(r0 + i, HID + f0)) =
                        make_uint4(aw[0], aw[1], aw[2], aw[3]);
                    i += 1;
                    ke[1] = ke[2];
                    ke[2] = ke[3];
                    ke[3] = ke[4];
                    deg = ke[1] - k1;
                    k1 = ke[1];
                };
                auto fetch = [&](uint4(&q)[GB], int k) {
#pragma unroll
                    for (int u = 0; u < GB; ++u)
                        if (k + u < kn) {
                            const int j = STAGED ? sn[k - ka + u] : nbr[k + u];
                            q[u] = qrow[(size_t)j * (2 * HID / 8)];
                        }
                };
                auto use = [&](const uint4(&q)[GB], int k) {
#pragma unroll
                    for (int u = 0; u < GB; ++u)
                        if (k + u < kn) {
                            while (k + u == k1) {
                                close();
                                open();
                            }
                            const float* ep = STAGED ? se + 3 * (k - ka + u) : e + 3 * (size_t)(k + u);
                            const f32x2 e0 = pair(ep[0], ep[0]), e1 = pair(ep[1], ep[1]),
                                        e2 = pair(ep[2], ep[2]);
                            const unsigned qw[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                // z = (p + c) + q + fma(C2, e2, fma(C0, e0, C1 e1))
                                const float2 z = unpair(
                                    add2(add2(pz[c], widen2(qw[c])),
                                         fma2(C2[c], e2, fma2(C0[c], e0, mul2(C1[c], e1)))));
                                acc[c] = add2(acc[c], pair(fmaxf(z.x, 0.f), fmaxf(z.y, 0.f)));
                            }
                        }
                };
                uint4 qa[GB], qb[GB];
                fetch(qa, ke[0]);
                open();
                for (int k = ke[0]; k < kn; k += GB) {
                    fetch(qb, k + GB);
                    use(qa, k);
                    k += GB;
                    if (k >= kn) break;
                    fetch(qa, k + GB);
                    use(qb, k);
                }
                while (i < 4) {
                    close();
                    if (i < 4) open();
                }
            };
            if (staged && here) gather(std::true_type{});
            else if (here) gather(std::false_type{});
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        fence_smem_async();
        fence_before();
        __syncthreads();
        if (*abort_flag) break;
        if (!ENC) {
            // v = U [h; agg]: 8 MMAs of K = 16 into columns 0..63
            if (tid == 0) {
                fence_after();
#pragma unroll
                for (int kk = 0; kk < 2 * HID / 16; ++kk)
                    mma(tbase, sdesc(xa + kk * 2 * LBO_X, SBO_X, LBO_X),
                        sdesc(ua + kk * 2 * LBO, SBO_U, LBO), idesc_bf16(TM, HID), kk > 0 ? 1u : 0u);
                commit(ubar);
            }
            pending = true;
            // meanwhile the next tile's edges: every warp has read this one's
            if (more) {
                tk0 = nk0;
                tk1 = nk1;
                pv = nv;
                stage();
            }
            // the warp goes on only as a whole (tcgen05.ld is warp-collective)
            if (!__all_sync(0xffffffffu, wait_parity(ubar, phase & 1))) {
                atomicExch(err, (int)CFD_ERR_BARRIER);
                *abort_flag = 1;
            } else {
                pending = false;
                phase += 1;
                fence_after();
                // h <- h + relu(v + u) on this thread's row, columns [32 half, +32)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    float a16[16];
                    tmem_ld16(tlane + 32 * half + 16 * c, a16);
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const int k0 = 32 * half + 16 * c + 8 * v;
                        uint4* xp = reinterpret_cast<uint4*>(Xs + x_off(erow, k0));
                        float h[8];
                        unpack8(*xp, h);
#pragma unroll
                        for (int i = 0; i < 8; ++i) h[i] = h[i] + fmaxf(a16[8 * v + i] + us[k0 + i], 0.f);
                        *xp = pack8(h);
                    }
                }
            }
            fence_smem_async();
            fence_before();
            __syncthreads();
            if (*abort_flag) break;
        }
        if (has_pq) {
            // P|Q = [A; B] h: 4 MMAs of K = 16 into columns 0..127
            if (tid == 0) {
                fence_after();
#pragma unroll
                for (int kk = 0; kk < HID / 16; ++kk)
                    mma(tbase, sdesc(xa + kk * 2 * LBO_X, SBO_X, LBO_X),
                        sdesc(wa + kk * 2 * LBO, SBO_W, LBO), idesc_bf16(TM, 2 * HID), kk > 0 ? 1u : 0u);
                commit(ubar);
            }
            pending = true;
            // meanwhile the tile's h rows go out, 4 rows per store (the last layer's h has no reader)
            const int r0 = 32 * q4 + 16 * half;
#pragma unroll
            for (int it = 0; it < 4; ++it) {
                const int r = r0 + 4 * it + sub;
                if (tb + r < n)
                    *reinterpret_cast<uint4*>(hb + (size_t)(tb + r) * HID + f0) =
                        *reinterpret_cast<const uint4*>(Xs + x_off(r, f0));
            }
            const bool ok = __all_sync(0xffffffffu, wait_parity(ubar, phase & 1));
            if (!ok) {
                atomicExch(err, (int)CFD_ERR_BARRIER);
                *abort_flag = 1;
            } else {
                pending = false;
                phase += 1;
                fence_after();
            }
            // P|Q rows into the tile's place (its MMAs are done; the pair of warps has read its h
            // rows), then out, 2 rows per store
            pair_sync(q4);
            unsigned char* st = Xs + PQ_BLK * q4;
            if (ok) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float v[16];
                    tmem_ld16(tlane + 64 * half + 16 * c, v);
                    uint4* op = reinterpret_cast<uint4*>(st + lane * PQ_ROW + 128 * half + 32 * c);
                    op[0] = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]),
                                       pack2(v[6], v[7]));
                    op[1] = make_uint4(pack2(v[8], v[9]), pack2(v[10], v[11]), pack2(v[12], v[13]),
                                       pack2(v[14], v[15]));
                }
            }
            pair_sync(q4);
#pragma unroll
            for (int it = 0; it < 8; ++it) {
                const int r = 16 * half + 2 * it + (lane >> 4), node = tb + 32 * q4 + r;
                if (node < n)
                    *reinterpret_cast<uint4*>(pq_out + (size_t)node * 2 * HID + 8 * (lane & 15)) =
                        *reinterpret_cast<const uint4*>(st + r * PQ_ROW + 16 * (lane & 15));
            }
        } else if (half == 0) {
            // decoder: y = W_out h + b_out on this thread's row
            const int node = tb + erow;
            float a[OUT];
#pragma unroll
            for (int o = 0; o < OUT; ++o) a[o] = wo[OUT * HID + o];
#pragma unroll 2
            for (int c = 0; c < HID / 8; ++c) {
                float h[8];
                unpack8(*reinterpret_cast<const uint4*>(Xs + x_off(erow, 8 * c)), h);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int o = 0; o < OUT; ++o) a[o] += wo[o * HID + 8 * c + i] * h[i];
            }
            if (node < n)
#pragma unroll
                for (int o = 0; o < OUT; ++o) y[(size_t)OUT * node + o] = a[o];
        }
        fence_before();
        __syncthreads();
        if (*abort_flag) break;
    }
    // what timed out or was left may still land: wait for it (bounded) before the memory goes
    if (tid == 0 && pending) wait_parity(ubar, phase & 1);
    if (spending) wait_parity(sbar, sphase & 1);
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase),
                     "r"(TMEM_COLS)
                     : "memory");
    }
}
}  // namespace tc

int infer_bf16(cudaStream_t st, const float* w, bf16* wb, bool* wb_valid, int n, const int* ptr,
               const int* nbr, const float* f, const float* e, bf16* hb, bf16* pqb, float* y,
               const int* gate, int* err) {
    if (!*wb_valid) {
        CFD_LAUNCH(k_to_bf16, blocks_for(N_PARAMS, 256), 256, 0, st, N_PARAMS, w, wb);
        *wb_valid = true;
    }
    int dev = 0, nsm = 1;
    CFD_CUDA(cudaGetDevice(&dev));
    CFD_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    bf16* pq[2] = {pqb, pqb + (size_t)n * 2 * HID};
    // tensor-core generation: tcgen05 unless CFD_MPNN_TC=0 (the mma.sync passes)
    const char* tce = getenv("CFD_MPNN_TC");
    if (!(tce && atoi(tce) == 0)) {
        static bool tc_attr = false;
        if (!tc_attr) {
            CFD_CUDA(cudaFuncSetAttribute(tc::k_infer_tc<true>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, tc::SMEM));
            CFD_CUDA(cudaFuncSetAttribute(tc::k_infer_tc<false>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, tc::SMEM));
            tc_attr = true;
        }
        const int ntile = (n + tc::TM - 1) / tc::TM;
        const int grid = std::max(1, std::min(ntile, 2 * nsm));
        CFD_LAUNCH(tc::k_infer_tc<true>, grid, tc::NTHR, tc::SMEM, st, n, 0, ptr, nbr, e, f, w,
                   (const bf16*)wb, 1, (const bf16*)nullptr, hb, pq[0], y, gate, err);
        for (int l = 0; l < LAYERS; ++l) {
            const int next = l + 1 < LAYERS ? 1 : 0;
            CFD_LAUNCH_CHAIN(tc::k_infer_tc<false>, grid, tc::NTHR, tc::SMEM, st, n, l, ptr, nbr, e,
                             f, w, (const bf16*)wb, next, (const bf16*)pq[l & 1], hb,
                             pq[(l + 1) & 1], y, gate, err);
        }
        return CFD_OK;
    }
    const size_t smem_enc = sizeof(bf16) * (2 * HID * HS + IW * 16 * HS) +
                            sizeof(float) * (HID * F_IN + HID);
    const size_t smem_layer = sizeof(bf16) * (HID * XS + 2 * HID * HS + IW * 16 * XS) +
                              sizeof(float) * (HID * E_F + 2 * HID);
    static bool attr_set = false;
    if (!attr_set) {
        CFD_CUDA(cudaFuncSetAttribute(k_infer_encode, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem_enc));
        CFD_CUDA(cudaFuncSetAttribute(k_infer_layer, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem_layer));
        attr_set = true;
    }
    const int ntile = (n + TILE - 1) / TILE;
    const int grid = std::min(ntile, 2 * nsm);  // resident blocks (registers, shared memory)
    CFD_LAUNCH(k_infer_encode, grid, 32 * IW, smem_enc, st, n, f, w, (const bf16*)wb, hb, pq[0],
               gate);
    for (int l = 0; l < LAYERS; ++l) {
        const int next = l + 1 < LAYERS ? 1 : 0;
        CFD_LAUNCH(k_infer_layer, grid, 32 * IW, smem_layer, st, n, l, ptr, nbr, e, w,
                   (const bf16*)wb, next, (const bf16*)pq[l & 1], hb, pq[(l + 1) & 1], y, gate);
    }
    return CFD_OK;
}

}  // namespace mpnn
}  // namespace cfd
