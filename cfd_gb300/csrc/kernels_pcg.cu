// kernels_pcg.cu — biCG (biconjGrad.f90:8-62) as one persistent cooperative kernel.
//
// The reference's solver is Jacobi-preconditioned CG with Dirichlet rows handled by
// overwrite and a 1e30 penalty; every vector operation is a separate OpenMP loop and the
// dots are OpenMP reductions.  Here the whole solve (both mesh-motion right-hand sides at
// once, sharing the matrix reads) is one launch: each iteration is three grid-wide passes
// separated by bounded grid barriers.
//   phase 1: x += alfa*p (deferred from the previous iteration), r -= alfa*y, z = r/diag,
//            partial sums of r.z (and of r.r under a relative stopping test)
//   phase 2: p_new = beta*p + z per row (biconjGrad.f90's vector update), a grid barrier,
//            then y = A.p_new, y(fix) = 1e30*p_new(fix), partial p.y
//   (the quotients z = r/diag use a reciprocal formed once per solve and two FMA
//   corrections, which give the division's bits: div_rcp)
// Every block folds the chunk partials itself in the fixed order of cfd_common.cuh, so
// all blocks hold bit-identical scalars and take the same branch.  With --fmad=false the
// iterates equal the CPU restatement's bit for bit.
//
// A block of 1024 threads takes a 1024-row chunk of the dots' order, one row per thread.
// ON_CHIP (no more chunks than SMs: up to 155,648 rows on 152 SMs): the row's x, r, p and y or
// z stay in the thread's registers for the whole solve and the matrix rows in shared memory
// (the first kEll entries; longer rows read the rest from global memory), so an iteration
// moves p alone through L2; the chunk's rows are dealt to the warps by length, so that a warp
// runs as many column steps as its rows have entries.  Otherwise a block walks over its
// chunks with the vectors in global memory, read by the thread that wrote them (p excepted).
// What bounds an iteration: the FP64 pipe (31 operations per row at 2 per clock and SM) and
// three barriers with two folds, which one warp per sum does alone: the chunk's products and
// the partials go from memory straight into the fixed tree, and the scalars' divisions are
// made once per block.  With 256-thread blocks (four rows per thread, vectors and matrix
// re-read, every thread dividing the scalars) an iteration took 32.1 us at 147,456 rows,
// 46.0 at 262,144 and 167 at 1,048,576; now 21.8, 43.9 and 145 us.
#include "cfd_kernels.cuh"

namespace cfd {

constexpr int kEll = 10;              // matrix entries per row kept in shared memory
constexpr int kPad = kChunk + 32;     // a chunk's products, one pad per 32
constexpr int kSortLen = 32;          // row-length classes of the deal
constexpr int kGroup = 4;             // chunks a block takes between two barriers of its own

// ------------------------------------------------------------------ barrier of one launch
// gb->arrive counts arrivals from zero; a waiter leaves when the count has reached `target`
// (compared modulo 2^32).  One hop: the last arrival itself releases the waiters.  false: the
// wait gave up after about `limit` polls or kWaitNs, or another wait has (gb->err is set).  The
// last block to leave a launch that did not fail clears the count for the next one (gb->gen
// counts the leavers), so that no clearing stands before each launch.  A failure leaves the count
// as it stood; launches that find err set do nothing, until the host has reported and cleared it.
// bar_clock, every 64 polls: when the wait began (0 before), or ~0 to give up; one copy, out of
// the iterations' instructions.
__device__ __noinline__ unsigned long long bar_clock(GridBar* gb, unsigned long long t0, bool over) {
    if (*(volatile const int*)&gb->err) return ~0ull;
    const unsigned long long now = globaltimer_ns();
    if (t0 == 0) t0 = now;
    if (!over && now - t0 <= kWaitNs) return t0;
    atomicExch(&gb->err, (int)CFD_ERR_BARRIER);
    return ~0ull;
}
__device__ __forceinline__ bool bar_arrive_wait(GridBar* gb, unsigned target,
                                                long long limit = kSpinLimit) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&gb->arrive) : "memory");
    unsigned long long t0 = 0;
    for (long long spins = 0;; ++spins) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&gb->arrive) : "memory");
        if ((int)(v - target) >= 0) return true;
        if ((spins & 63) == 63 && (t0 = bar_clock(gb, t0, spins > limit)) == ~0ull) return false;
    }
}

// A chunk's cnt products in shared memory (pad32) -> their sum in the dots' order, by one
// warp.  A whole chunk takes the branch-free form, whose 32 loads and eight chains of adds
// overlap.  One copy for all passes (noinline): an iteration runs each pass once, so inlined
// copies would be fetched anew.
__device__ __noinline__ double chunk_sum(const double* q, int cnt) {
    if (cnt == kChunk)
        return warp_tree256([&](int t) {
            return ((q[pad32(t)] + q[pad32(t + 256)]) + q[pad32(t + 512)]) + q[pad32(t + 768)];
        });
    return warp_tree256([&](int t) {
        double acc = t < cnt ? q[pad32(t)] : 0.0;
#pragma unroll
        for (int k = 1; k < 4; ++k)
            if (t + 256 * k < cnt) acc = acc + q[pad32(t + 256 * k)];
        return acc;
    });
}

// The nc chunk partials -> their fold (256 lanes with stride 256, then the tree), by one warp; the
// loads are clamped, not branched over, so that a lane's eight go out together
__device__ __noinline__ double chunk_fold(const double* part, long nc) {
    const int lane = threadIdx.x & 31, t = 32 * (lane >> 2) + (lane & 3);
    double acc[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const long c = t + 4 * u;
        acc[u] = __ldcg(part + min(c, nc - 1));
        if (c >= nc) acc[u] = 0.0;
    }
    for (long base = 256; base < nc; base += 512) {
        double v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u)
            v[u] = __ldcg(part + min(base + t + 4 * (u & 7) + 256 * (u >> 3), nc - 1));
#pragma unroll
        for (int u = 0; u < 16; ++u)
            if (base + t + 4 * (u & 7) + 256 * (u >> 3) < nc) acc[u & 7] = acc[u & 7] + v[u];
    }
    return warp_tree256([&](int x) { return acc[(x - t) >> 2]; });
}

// Row i of A times the vectors of the ns solves, the row read from global memory in batches
// (a batch's columns and values, then its gathers, go out together); sums in column order.
// FIXC: also the sums over the Dirichlet columns only, the product with x_D, the vector that
// is v on the Dirichlet rows and 0 elsewhere (a skipped term adds +0, which leaves a sum
// that starts at +0 unchanged).
template <bool FIXC>
__device__ __forceinline__ void row_products(const PcgArgs& a, int j0, int j1, const double* v0,
                                             const double* v1, double (&dot)[2],
                                             double (&dfix)[2]) {
    constexpr int B = 4;
    double d0 = 0.0, d1 = 0.0, f0 = 0.0, f1 = 0.0;
    for (int jb = j0; jb < j1; jb += B) {
        int c[B];
        double m[B], x0[B], x1[B];
        bool fx[B];
#pragma unroll
        for (int u = 0; u < B; ++u)
            if (jb + u < j1) {
                c[u] = a.col[jb + u];
                m[u] = a.val[jb + u];
            }
#pragma unroll
        for (int u = 0; u < B; ++u)
            if (jb + u < j1) {
                if (v0) x0[u] = v0[c[u]];
                if (v1) x1[u] = v1[c[u]];
                if (FIXC) fx[u] = a.isfix[c[u]] != 0;
            }
#pragma unroll
        for (int u = 0; u < B; ++u)
            if (jb + u < j1) {
                if (v0) {
                    const double t = m[u] * x0[u];
                    d0 = d0 + t;
                    if (FIXC && fx[u]) f0 = f0 + t;
                }
                if (v1) {
                    const double t = m[u] * x1[u];
                    d1 = d1 + t;
                    if (FIXC && fx[u]) f1 = f1 + t;
                }
            }
    }
    dot[0] = d0;
    dot[1] = d1;
    dfix[0] = f0;
    dfix[1] = f1;
}

// Which partials a pass's sums go to: slot j in byte j, 2 * buffer + solve
__device__ __forceinline__ int slot_at(unsigned code, int j) { return (int)(code >> (8 * j)) & 0xff; }

// What the block's threads share; prod[g][j]: the products of the group's chunk g, sum j
template <int G>
struct PcgShared {
    double prod[G][4][kPad];
    double alfa[2], beta[2], err_new[2], err_old[2], rold[2], rr[2], thr[2], ref2[2];
    int act[2], pend[2], done[2], last[2], fail;
    int hist[kSortLen];
    unsigned short perm[kChunk];
};

template <bool ON_CHIP>
__global__ void __launch_bounds__(kChunk, 1) k_pcg_fp64(PcgArgs a) {
    extern __shared__ __align__(16) unsigned char pcg_smem[];
    constexpr int G = ON_CHIP ? 1 : kGroup;
    typedef PcgShared<G> Shared;
    Shared& s = *reinterpret_cast<Shared*>(pcg_smem);
    double* ellv = reinterpret_cast<double*>(pcg_smem + sizeof(Shared));  // [kEll][kChunk]
    int* ellc = reinterpret_cast<int*>(ellv + kEll * kChunk);
    const int t = threadIdx.x, wp = t >> 5, lane = t & 31;
    const int n = a.n, ns = a.nsolve;
    const long nc = ((long)n + kChunk - 1) / kChunk;
    const unsigned nb = gridDim.x;
    unsigned target = 0;
    const bool rel = a.tol_mode != CFD_BICG_TOL_ABS;   // r.r per iteration
    const bool relb = a.tol_mode == CFD_BICG_TOL_REL;  // ||b - A.x_D|| as reference
    // after a barrier of an earlier launch gave up; one thread reads it, for the whole block
    if (__syncthreads_or(t == 0 && *(volatile const int*)&a.bar->err != 0)) return;
    if (t == 0) s.fail = 0;

    auto leave = [&] {  // one thread; the block waits no more
        if (atomicAdd(&a.bar->gen, 1u) == nb - 1) {
            a.bar->arrive = 0u;
            a.bar->gen = 0u;
        }
    };
    // every thread's global writes before, every thread's reads after
    auto grid_sync = [&]() -> bool {
        __syncthreads();
        target += nb;
        if (t == 0 && !bar_arrive_wait(a.bar, target)) s.fail = 1;
        __syncthreads();
        return s.fail == 0;
    };
    // the sums of the group of chunks c, c + nb, ... (slot j of chunk g = prod[g][j], into the
    // partials code names), one warp per sum
    auto chunk_sums = [&](long c, int m, unsigned code) {
        __syncthreads();
        const int g = wp >> 2, j = wp & 3;
        const long cg = c + (long)g * nb;
        if (g < G && j < m && cg < nc) {
            const double v = chunk_sum(s.prod[g][j], (int)min((long)kChunk, n - cg * kChunk));
            const int q = slot_at(code, j);
            if (lane == 0) a.part[q * nc + cg] = v;
        }
        __syncthreads();  // several warps' partials precede one arrival; prod may be refilled
    };
    // the grid's folds of the same slots: warp j arrives for slot j, waits, folds, and hands
    // the sum to `use` in lane 0; the other warps run `meanwhile`, warps 0..m-1 after their
    // folds
    auto fold_sums = [&](int m, unsigned code, auto use, auto meanwhile) -> bool {
        target += nb * (unsigned)m;
        if (wp < m) {
            int ok = 1;
            if (lane == 0) ok = bar_arrive_wait(a.bar, target) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            __syncwarp();  // lane 0's acquire comes before every lane's reads (a shuffle orders none)
            if (ok) {
                const int q = slot_at(code, wp);
                const double v = chunk_fold(a.part + q * nc, nc);
                if (lane == 0) use(wp, q & 1, v);
            } else if (lane == 0) {
                s.fail = 1;
            }
        }
        meanwhile();
        __syncthreads();
        return s.fail == 0;
    };
    auto nothing = [] {};

    // copy1 (biconjGrad.f90:28): x(fix) = x_fix
    for (int k = blockIdx.x * kChunk + t; k < a.nfix; k += gridDim.x * kChunk)
        for (int q = 0; q < ns; ++q) a.x[q][a.fix_node[k]] = 1.0 * a.fixval[q][a.fix_src[k]];

    // ON_CHIP: the thread's row (by length class within the chunk) and its matrix entries
    long row = -1;   // the thread's row; -1: none
    int slot = 0;    // its position in the chunk (the dots' order)
    int len = 0, jx = 0;
    bool fx = false;
    double d = 1.0, rd = 1.0;
    double xr[2] = {0.0, 0.0}, rr_[2] = {0.0, 0.0}, pr[2] = {0.0, 0.0}, yz[2] = {0.0, 0.0};
    if (ON_CHIP) {
        const long i = (long)blockIdx.x * kChunk + t;
        int key = 0;
        if (i < n && !a.isfix[i])  // row pointers that descend: an empty row, as in the row loops
            key = max(0, min(a.rowptr[i + 1] - a.rowptr[i], kSortLen - 1));
        if (t < kSortLen) s.hist[t] = 0;
        __syncthreads();
        if (i < n) atomicAdd(&s.hist[key], 1);
        __syncthreads();
        if (wp == 0) {  // exclusive prefix of the 32 classes
            const int v = s.hist[lane];
            int x = v;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, off);
                if (lane >= off) x += y;
            }
            s.hist[lane] = x - v;
        }
        __syncthreads();
        if (i < n) s.perm[atomicAdd(&s.hist[key], 1)] = (unsigned short)t;
        __syncthreads();
        if (i < n) {  // as many threads as rows: thread t takes the t-th of the deal
            slot = s.perm[t];
            row = (long)blockIdx.x * kChunk + slot;
            fx = a.isfix[row] != 0;
            d = a.diag[row];
            rd = 1.0 / d;
            if (!fx) {
                jx = a.rowptr[row];
                len = a.rowptr[row + 1] - jx;
#pragma unroll
                for (int u = 0; u < kEll; ++u)
                    if (u < len) {
                        ellv[u * kChunk + t] = a.val[jx + u];
                        ellc[u * kChunk + t] = a.col[jx + u];
                    }
            }
        }
    }
    // ON_CHIP row product with v (global memory), in column order
    auto chip_row = [&](const double* v) {
        double dot = 0.0, g[kEll];
#pragma unroll
        for (int u = 0; u < kEll; ++u)
            if (u < len) g[u] = v[ellc[u * kChunk + t]];
#pragma unroll
        for (int u = 0; u < kEll; ++u)
            if (u < len) dot = dot + ellv[u * kChunk + t] * g[u];
        for (int u = kEll; u < len; ++u) dot = dot + a.val[jx + u] * v[a.col[jx + u]];
        return dot;
    };
    if (a.nfix > 0 && !grid_sync()) return;

    // y = A.x; y(fix) = 1e30*x(fix); r = -1*y + b; r(fix) = 0; r.r   (:138-144)
    // CFD_BICG_TOL_REL also forms b - A.x_D (0 on the Dirichlet rows) and its square sum
    // slots: r.r of the solves (buffer 0), then (relb) the reference norms (buffer 2)
    const int m0 = (relb ? 2 : 1) * ns;
    const unsigned code0 = ns > 1 ? 0x05040100u : 0x00000400u;
    auto first_row = [&](long i, int sl, int g) {
        const bool f = a.isfix[i] != 0;
        double dot[2] = {0.0, 0.0}, df[2] = {0.0, 0.0};
        if (!f) {
            const int j0 = a.rowptr[i], j1 = a.rowptr[i + 1];
            const double* v1 = ns > 1 ? a.x[1] : nullptr;
            if (relb) row_products<true>(a, j0, j1, a.x[0], v1, dot, df);
            else row_products<false>(a, j0, j1, a.x[0], v1, dot, df);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (q >= ns) break;
            const double xi = a.x[q][i];
            const double yi = f ? 1.0e30 * xi : dot[q];
            const double bi = a.b[q] ? a.b[q][i] : 0.0;
            double ri = -1.0 * yi + bi;
            if (f) ri = 0.0;
            if (ON_CHIP) {
                xr[q] = xi;
                rr_[q] = ri;
            } else {
                a.r[q][i] = ri;
            }
            s.prod[g][q][pad32(sl)] = ri * ri;
            if (relb) {
                double ei = -1.0 * df[q] + bi;
                if (f) ei = 0.0;
                s.prod[g][ns + q][pad32(sl)] = ei * ei;
            }
        }
    };
    // for (chunk groups) { rows; sums }: row(i, position in the chunk, chunk of the group)
    auto rows_and_sums = [&](int m, unsigned code, auto on_row) {
        if (ON_CHIP) {
            if (row >= 0) on_row(row, slot, 0);
            chunk_sums(blockIdx.x, m, code);
        } else {
            for (long c = blockIdx.x; c < nc; c += (long)G * nb) {
#pragma unroll 2
                for (int g = 0; g < G; ++g) {
                    const long i = (c + (long)g * nb) * kChunk + t;
                    if (i < n) on_row(i, t, g);
                }
                chunk_sums(c, m, code);
            }
        }
    };
    rows_and_sums(m0, code0, first_row);
    if (!fold_sums(m0, code0,
                   [&](int j, int q, double v) {
                       if (j < ns) s.rr[q] = v;
                       else s.ref2[q] = v;
                   },
                   nothing))
        return;
    if (t < ns) {
        const double rr = s.rr[t];
        bool done;
        if (rel) {
            const double ref2 = relb ? s.ref2[t] : rr;
            s.ref2[t] = ref2;
            s.thr[t] = (a.tol * a.tol) * ref2;
            done = rr <= s.thr[t];
        } else {
            done = rr < a.tol;
        }
        s.done[t] = done;
        s.pend[t] = !done;
        s.last[t] = 0;
        if (done && blockIdx.x == 0) {
            a.iters_out[t] = 0;
            a.rz_out[t] = rr;
            a.conv_out[t] = 1;
            if (a.relres_out)
                a.relres_out[t] = (rel && s.ref2[t] > 0.0) ? sqrt(rr / s.ref2[t]) : 0.0;
        }
    }
    __syncthreads();
    bool done[2];
    done[0] = s.done[0] != 0;
    done[1] = ns < 2 || s.done[1] != 0;
    if (done[0] && done[1]) {
        if (t == 0) leave();
        return;
    }

    // the slots of the active solves' sums in buffer ba, then (two) in buffer bb
    auto slots = [&](bool on0, bool on1, bool two, unsigned ba, unsigned bb, unsigned& code) {
        const unsigned one = on0 ? (on1 ? 0x0100u + 0x0202u * ba : 2u * ba) : 2u * ba + 1u;
        const int m = (on0 ? 1 : 0) + (on1 ? 1 : 0);
        code = one;
        if (!two) return m;
        const unsigned sec = on0 ? (on1 ? 0x0100u + 0x0202u * bb : 2u * bb) : 2u * bb + 1u;
        code |= sec << (8 * m);
        return 2 * m;
    };
    unsigned code = 0;

    // p = r/diag; err_new = r.p   (:146-147)
    {
        const int m = slots(!done[0], !done[1], false, 1, 0, code);
        rows_and_sums(m, code, [&](long i, int sl, int g) {
            double di = d, rdi = rd;
            if (!ON_CHIP) {
                di = a.diag[i];
                rdi = 1.0 / di;
                a.rdiag[i] = rdi;
            }
            int j = 0;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (done[q]) continue;
                const double ri = ON_CHIP ? rr_[q] : a.r[q][i];
                const double pi = div_rcp(ri, di, rdi);
                a.p[q][0][i] = pi;
                if (ON_CHIP) pr[q] = pi;
                s.prod[g][j++][pad32(sl)] = ri * pi;
            }
        });
        // p of every block is in place too: the arrivals follow the block's writes of p
        // (__syncthreads in chunk_sums, the release at the arrival)
        if (!fold_sums(m, code, [&](int, int q, double v) { s.err_new[q] = v; }, nothing)) return;
    }

    // y = A.p; y(fix) = 1e30*p(fix); py = p.y; alfa = err_new/py   (:148-152), for the solves
    // with on[q]; x = alfa*p + x (:153) is applied in the next phase 1
    int k = 0;
    auto product = [&](bool on0, bool on1) -> bool {
        const int m = slots(on0, on1, false, 0, 0, code);
        rows_and_sums(m, code, [&](long i, int sl, int g) {
            int j = 0;
            if (ON_CHIP) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (!(q ? on1 : on0)) continue;
                    const double yi = fx ? 1.0e30 * pr[q] : chip_row(a.p[q][0]);
                    yz[q] = yi;
                    s.prod[0][j++][pad32(sl)] = pr[q] * yi;
                }
            } else {
                const bool f = a.isfix[i] != 0;
                double dot[2] = {0.0, 0.0}, df[2];
                if (!f)
                    row_products<false>(a, a.rowptr[i], a.rowptr[i + 1],
                                        on0 ? a.p[0][0] : nullptr, on1 ? a.p[1][0] : nullptr, dot,
                                        df);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (!(q ? on1 : on0)) continue;
                    const double pi = a.p[q][0][i];
                    const double yi = f ? 1.0e30 * pi : dot[q];
                    a.y[q][i] = yi;
                    s.prod[g][j++][pad32(sl)] = pi * yi;
                }
            }
        });
        return fold_sums(m, code,
                         [&](int, int q, double py) {
                             const double e = s.err_new[q];
                             s.alfa[q] = e / py;
                             s.err_old[q] = e;
                             s.pend[q] = 1;
                             s.last[q] = k;
                             s.act[q] =
                                 (rel ? s.rr[q] > s.thr[q] : fabs(e) > a.tol) && k < a.maxit;
                         },
                         nothing);
    };
    if (!product(!done[0], !done[1])) return;

    while (true) {  // :156-170
        const bool act[2] = {!done[0] && s.act[0] != 0, !done[1] && s.act[1] != 0};
        if (!act[0] && !act[1]) break;
        k = k + 1;
        // phase 1; 1/err_old for beta's quotient is formed beside it by an idle thread
        {
            const bool pend[2] = {!done[0] && s.pend[0] != 0, !done[1] && s.pend[1] != 0};
            const double alfa[2] = {s.alfa[0], s.alfa[1]};
            const int m = slots(act[0], act[1], rel, 1, 2, code);
            const int na = (act[0] ? 1 : 0) + (act[1] ? 1 : 0);
            if (t >= kChunk - 2) s.rold[t - (kChunk - 2)] = 1.0 / s.err_old[t - (kChunk - 2)];
            rows_and_sums(m, code, [&](long i, int sl, int g) {
                double di = d, rdi = rd;
                if (!ON_CHIP) {
                    di = a.diag[i];
                    rdi = a.rdiag[i];
                }
                int j = 0;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (!ON_CHIP && pend[q]) a.x[q][i] = alfa[q] * a.p[q][0][i] + a.x[q][i];
                    if (!act[q]) continue;
                    const double ri = (-alfa[q]) * (ON_CHIP ? yz[q] : a.y[q][i]) +
                                      (ON_CHIP ? rr_[q] : a.r[q][i]);
                    const double zi = div_rcp(ri, di, rdi);
                    if (ON_CHIP) {
                        rr_[q] = ri;
                        yz[q] = zi;
                    } else {
                        a.r[q][i] = ri;
                        a.z[q][i] = zi;
                    }
                    s.prod[g][j][pad32(sl)] = ri * zi;
                    if (rel) s.prod[g][na + j][pad32(sl)] = ri * ri;
                    ++j;
                }
            });
            if (!fold_sums(m, code,
                           [&](int j, int q, double v) {
                               if (j >= na) {
                                   s.rr[q] = v;
                                   return;
                               }
                               s.err_new[q] = v;
                               s.beta[q] = div_rcp(v, s.err_old[q], s.rold[q]);
                           },
                           [&] {  // the deferred x update, under the barrier
                               if (ON_CHIP && row >= 0)
#pragma unroll
                                   for (int q = 0; q < 2; ++q)
                                       if (pend[q]) xr[q] = alfa[q] * pr[q] + xr[q];
                           }))
                return;
            if (t < 2) {  // read again by the next phase 1 or the end, behind barriers
                s.pend[t] = 0;
                if (!(t ? act[1] : act[0])) s.act[t] = 0;
            }
        }
        // phase 2a: p_new = beta p + z, once per row (the SpMV below reads it; forming it
        // inside every row's column loop would cost two FP64 operations per entry)
        {
            const double beta[2] = {s.beta[0], s.beta[1]};
            if (ON_CHIP) {
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (act[q] && row >= 0) {
                        pr[q] = beta[q] * pr[q] + yz[q];
                        a.p[q][0][row] = pr[q];
                    }
            } else {
                for (long c = blockIdx.x; c < nc; c += gridDim.x) {
                    const long i = c * kChunk + t;
                    if (i < n)
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            if (act[q]) a.p[q][0][i] = beta[q] * a.p[q][0][i] + a.z[q][i];
                }
            }
        }
        if (!grid_sync()) return;
        // phase 2b: y = A p_new, y(fix) = 1e30 p_new(fix), p.y, alfa
        if (!product(act[0], act[1])) return;
    }
    // the last deferred x update
    {
        const bool pend[2] = {!done[0] && s.pend[0] != 0, !done[1] && s.pend[1] != 0};
        const double alfa[2] = {s.alfa[0], s.alfa[1]};
        if (ON_CHIP) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (row >= 0 && !done[q])
                    a.x[q][row] = pend[q] ? alfa[q] * pr[q] + xr[q] : xr[q];
        } else {
            for (long c = blockIdx.x; c < nc; c += gridDim.x) {
                const long i = c * kChunk + t;
                if (i < n)
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        if (pend[q]) a.x[q][i] = alfa[q] * a.p[q][0][i] + a.x[q][i];
            }
        }
    }
    if (t == 0) leave();
    if (blockIdx.x == 0 && t < ns && !s.done[t]) {
        a.iters_out[t] = s.last[t];
        a.rz_out[t] = fabs(s.err_old[t]);
        a.conv_out[t] = (rel ? s.rr[t] > s.thr[t] : fabs(s.err_old[t]) > a.tol) ? 0 : 1;
        if (a.relres_out)
            a.relres_out[t] = (rel && s.ref2[t] > 0.0) ? sqrt(s.rr[t] / s.ref2[t]) : 0.0;
    }
}

// One solve on the current device (a.bar: zeroed once, or left so by the last launch): ON_CHIP when
// the chunks fit the SMs one each
cudaError_t launch_pcg_fp64(cudaStream_t st, PcgArgs a) {
    int dev = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const long nc = ((long)a.n + kChunk - 1) / kChunk;
    const bool chip = nc <= nsm;
    const int smem = chip ? (int)sizeof(PcgShared<1>) + kEll * kChunk * 12 : (int)sizeof(PcgShared<kGroup>);
    const void* fn = chip ? (const void*)k_pcg_fp64<true> : (const void*)k_pcg_fp64<false>;
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess)
        return e;
    const unsigned grid = (unsigned)(chip ? nc : nsm);
    void* args[] = {&a};
    e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kChunk), args, (size_t)smem, st);
    if (e == cudaSuccess) g_launches.fetch_add(1, std::memory_order_relaxed);
    return e;
}

// CFD_GUESS_EXTRAPOLATED: the solves start from the last two increments extrapolated to
// this step.  A solve's unknown is the step's mesh increment, the mean mesh velocity over the
// step times DTMIN; with that velocity linear in time through the last two steps' midpoints,
//     x = c1 x_{n-1} + c2 x_{n-2},  h = (dt_n + dt1) / (dt1 + dt2),
//     c1 = dt_n / dt1 (1 + h),  c2 = -(dt_n / dt2) h
// on the free rows (x_{n-1} is the previous solution, still in x), in the oracle's operation
// order (--fmad=false: the same bits); x_{n-1} is kept as the next step's x_{n-2}; with fewer
// than two kept the guess stays x_{n-1}.  hist[3..5] = (c1, c2, two kept) from guess_history: a
// division is ten operations of the FP64 pipe, and a thread takes a node or two.  The fixed
// rows are left to the Dirichlet values (set before, or by the solve).  The float shadow and,
// under the relative tests, the hi/lo split (mixed form) follow x.
__global__ void k_guess_extrapolate(PcgArgs a, const double* __restrict__ hist,
                                    double* __restrict__ xprev0, double* __restrict__ xprev1) {
    const double c1 = hist[3], c2 = hist[4];
    const bool two = hist[5] != 0.0;
    // two rows and both solves' loads go out together
    const long step = (long)gridDim.x * blockDim.x;
    for (long i0 = blockIdx.x * (long)blockDim.x + threadIdx.x; i0 < a.n; i0 += 2 * step) {
        double x[2][2], xp[2][2];
        bool fx[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const long i = min(i0 + u * step, (long)a.n - 1);
            fx[u] = a.isfix[i] != 0;
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (s < a.nsolve) {
                    x[u][s] = a.x[s][i];
                    xp[u][s] = (s ? xprev1 : xprev0)[i];
                }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const long i = i0 + u * step;
            if (i >= a.n) break;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                if (s >= a.nsolve) break;
                const double x1 = x[u][s];
                double xn = x1;
                if (!fx[u]) {
                    if (two) {
                        xn = c1 * x1 + c2 * xp[u][s];
                        a.x[s][i] = xn;
                        if (a.xf[s]) a.xf[s][i] = d2f_trunc(xn);
                    }
                    (s ? xprev1 : xprev0)[i] = x1;
                }
                if (a.xs[s]) {  // the precise product's operand (mixed form, relative tests)
                    float hi, lo;
                    split_bits(xn, hi, lo);
                    a.xs[s][i] = make_float2(hi, lo);
                }
            }
        }
    }
}

// before k_guess_extrapolate: guess_history, by one thread (the mixed form's k_motion_tail
// has it done beside the motion)
__global__ void k_guess_extrapolate_hist(const double* __restrict__ dtn_p,
                                         double* __restrict__ hist) {
    if (blockIdx.x == 0 && threadIdx.x == 0) guess_history(*dtn_p, hist);
}

// div_rcp and div_rcp2 against the division x / d over n input pairs, a quarter of each kind: raw
// 64-bit patterns for both (splitmix64: every exponent and sign, subnormals, infinities, NaNs);
// both of magnitude 2^-60 .. 2^60; x = d * m for a random significand m moved by up to +-2^12
// ulps (quotients next to binade edges and to halfway cases); the ends of the range that the
// short forms take (exponents 200 and 1800, 800 apart, one more and one less) and x = +-0.
// Counts the pairs whose results differ in any bit (NaNs count as equal).
__device__ __forceinline__ unsigned long long splitmix(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__global__ void k_selftest_divrcp(long long n, unsigned long long seed,
                                  unsigned long long* __restrict__ bad) {
    unsigned long long local = 0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
        const unsigned long long z1 = splitmix(seed + (unsigned long long)i * 0x9e3779b97f4a7c15ull);
        const unsigned long long z2 = splitmix(z1 + 0x632be59bd9b4e019ull);
        unsigned long long bx = z1, bd = z2;
        const int kind = (int)(i % 4);
        if (kind == 1) {
            bx = (z1 & 0x800fffffffffffffull) | ((963ull + (z1 >> 52) % 121ull) << 52);
            bd = (z2 & 0x800fffffffffffffull) | ((963ull + (z2 >> 52) % 121ull) << 52);
        } else if (kind == 2) {
            bd = (z2 & 0x800fffffffffffffull) | ((993ull + (z2 >> 52) % 61ull) << 52);
            const double m = __longlong_as_double((long long)((z1 & 0x000fffffffffffffull) |
                                                              (1023ull << 52)));
            const long long b = __double_as_longlong(__longlong_as_double((long long)bd) * m);
            bx = (unsigned long long)(b + ((long long)(z1 >> 52 & 0x1fffull) - 4096));
        } else if (kind == 3) {
            const int end[8] = {0, 199, 200, 201, 1023, 1799, 1800, 1801};
            const int apart[8] = {-801, -800, -799, 0, 799, 800, 801, 0};
            const int ed = end[z2 >> 52 & 7], k = (int)(z1 >> 52 & 7);
            const int ex = k == 3 ? end[z1 >> 55 & 7] : min(max(ed + apart[k], 0), 2046);
            bd = (z2 & 0x800fffffffffffffull) | ((unsigned long long)ed << 52);
            bx = z1 & 0x8000000000000000ull;
            if (k < 7) bx = (z1 & 0x800fffffffffffffull) | ((unsigned long long)ex << 52);
        }
        const double x = __longlong_as_double((long long)bx), d = __longlong_as_double((long long)bd);
        const double y = 1.0 / d;
        const double a = div_rcp(x, d, y), b = x / d;
        const double c = div_rcp2(x, d, y, rcp_lo(d, y));
        const bool nan = a != a && b != b && c != c;
        if ((__double_as_longlong(a) != __double_as_longlong(b) ||
             __double_as_longlong(c) != __double_as_longlong(b)) && !nan)
            ++local;
    }
    if (local) atomicAdd(bad, local);
}

cudaError_t launch_selftest_divrcp(long long n, unsigned long long seed, unsigned long long* bad) {
    k_selftest_divrcp<<<152 * 8, 256>>>(n, seed, bad);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

// Failure-detection self-test of the mixed solve's grid barrier and the mbarrier wait (one block):
// a grid barrier that expects a second block that never comes, and an mbarrier nothing arrives
// on.  Both give up after `limit` polls; out[0] = the barrier's error word, out[1] =
// CFD_ERR_BARRIER when the mbarrier wait gave up (0 if it completed).
__global__ void k_selftest_waits(GridBar* gb, int* out, long long limit) {
    __shared__ __align__(8) unsigned long long bar;
    grid_barrier(gb, 2u, limit);
    if (threadIdx.x == 0) {
        const unsigned ubar = (unsigned)__cvta_generic_to_shared(&bar);
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ubar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        out[1] = mbar_wait_bounded(ubar, 0u, limit) ? 0 : (int)CFD_ERR_BARRIER;
        out[0] = gb->err;
    }
}

// The same of the FP64 solve's barrier: *out = the barrier's error word when the wait for a second
// arrival that never comes gave up, 0 if it did not.
__global__ void k_selftest_solve_wait(GridBar* gb, int* out, long long limit) {
    if (threadIdx.x == 0) *out = bar_arrive_wait(gb, 2u, limit) ? 0 : gb->err;
}

}  // namespace cfd
