// Block vectors: up to kBlkMax right-hand sides solved together (multi-RHS PCG with
// the AMG V-cycle).
//
// A block vector holds the ld columns interleaved per row (entry (i, c) at i*ld + c,
// ld even, columns beyond the caller's zero), in every vector of the solve, so a
// gather of one matrix entry is one run of 8*ld bytes and each matrix entry read
// serves all columns.  A thread owns one row and one pair of columns (16-byte loads);
// the ld/2 threads of a row read the same entry (one broadcast request) and
// neighbouring pairs of the gathered row.
//
// Sums run in CSR order per column (row split into W interleaved parts, added in
// order, where a level has too few rows to fill the GPU).  Covered: V-cycle, Jacobi
// smoothing (any n1, n2, omega), FP64, 1x1 or dense-inverse coarsest solve; anything
// else is applied column by column by the caller.
//
// Measured, 32 right-hand sides on a 64^3 Poisson system: groups of 8 columns, one
// thread per row with 8 accumulators and conversions to and from the block layout
// around every cycle, 55.6 ms (120 launches and 2 ms an iteration; a warp's 16-byte
// load of 32 separate rows is 32 lookups); this layout 25.1 ms.
#include "cycle.cuh"

#include <algorithm>

namespace lab
{
    constexpr int kBlkNT = 256;

    __device__ __forceinline__ double2 ld2(const double* p)
    {
        return __ldg(reinterpret_cast<const double2*>(p));
    }
    __device__ __forceinline__ void st2(double* p, double2 v)
    {
        *reinterpret_cast<double2*>(p) = v;
    }
    __device__ __forceinline__ double2 mul2(double a, double2 v)
    {
        return {a * v.x, a * v.y};
    }

    // ------------------------------------------------------------ block ops
    // Same formulas as op_pre0 / op_jacobi / op_res / op_prolong / op_restrict, on one
    // pair of columns.  at: the pair's offset in row i.
    struct bop_pre0
    {
        static constexpr bool kDot = false;
        const double* __restrict__ b;
        const double* __restrict__ invd;
        double omega;
        double* __restrict__ x;
        double* __restrict__ r;
        struct pre_t
        {
            double2 b;
            double  invd;
        };
        __device__ __forceinline__ pre_t pre(int i, size_t at) const
        {
            return {ld2(b + at), __ldg(invd + i)};
        }
        __device__ __forceinline__ double2 gather(int c, size_t at) const
        {
            return mul2(omega, mul2(__ldg(invd + c), ld2(b + at)));
        }
        __device__ __forceinline__ double2 finish(size_t at, double2 s, const pre_t& p) const
        {
            st2(x + at, mul2(omega, mul2(p.invd, p.b)));
            st2(r + at, {p.b.x - s.x, p.b.y - s.y});
            return {0.0, 0.0};
        }
    };

    template <bool DOT>
    struct bop_jacobi
    {
        static constexpr bool kDot = DOT; // (y, b) per column
        const double* __restrict__ x;
        const double* __restrict__ b;
        const double* __restrict__ invd;
        double omega;
        double* __restrict__ y;
        struct pre_t
        {
            double2 x, b;
            double  invd;
        };
        __device__ __forceinline__ pre_t pre(int i, size_t at) const
        {
            return {ld2(x + at), ld2(b + at), __ldg(invd + i)};
        }
        __device__ __forceinline__ double2 gather(int, size_t at) const
        {
            return ld2(x + at);
        }
        __device__ __forceinline__ double2 finish(size_t at, double2 s, const pre_t& p) const
        {
            const double2 v{p.x.x + omega * (p.invd * (p.b.x - s.x)),
                            p.x.y + omega * (p.invd * (p.b.y - s.y))};
            st2(y + at, v);
            return {v.x * p.b.x, v.y * p.b.y};
        }
    };

    struct bop_res
    {
        static constexpr bool kDot = false;
        const double* __restrict__ x;
        const double* __restrict__ b;
        double* __restrict__ r;
        using pre_t = double2;
        __device__ __forceinline__ pre_t pre(int, size_t at) const
        {
            return ld2(b + at);
        }
        __device__ __forceinline__ double2 gather(int, size_t at) const
        {
            return ld2(x + at);
        }
        __device__ __forceinline__ double2 finish(size_t at, double2 s, const pre_t& p) const
        {
            st2(r + at, {p.x - s.x, p.y - s.y});
            return {0.0, 0.0};
        }
    };

    // y = x + P e
    struct bop_prolong
    {
        static constexpr bool kDot = false;
        const double* __restrict__ e;
        const double* __restrict__ x;
        double* __restrict__ y;
        using pre_t = double2;
        __device__ __forceinline__ pre_t pre(int, size_t at) const
        {
            return ld2(x + at);
        }
        __device__ __forceinline__ double2 gather(int, size_t at) const
        {
            return ld2(e + at);
        }
        __device__ __forceinline__ double2 finish(size_t at, double2 s, const pre_t& p) const
        {
            st2(y + at, {p.x + s.x, p.y + s.y});
            return {0.0, 0.0};
        }
    };

    // y = R r; with x0, also the coarse level's first sweep x0 = omega D_c^-1 y
    struct bop_restrict
    {
        static constexpr bool kDot = false;
        const double* __restrict__ r;
        double* __restrict__ y;
        const double* __restrict__ invd_c;
        double omega;
        double* __restrict__ x0;
        using pre_t = double;
        __device__ __forceinline__ pre_t pre(int i, size_t) const
        {
            return x0 ? __ldg(invd_c + i) : 0.0;
        }
        __device__ __forceinline__ double2 gather(int, size_t at) const
        {
            return ld2(r + at);
        }
        __device__ __forceinline__ double2 finish(size_t at, double2 s, const pre_t& p) const
        {
            st2(y + at, s);
            if(x0)
                st2(x0 + at, mul2(omega, mul2(p, s)));
            return {0.0, 0.0};
        }
    };

    // q = A p with (p, q) per column
    struct bop_spmv_dot
    {
        static constexpr bool kDot = true;
        const double* __restrict__ p;
        double* __restrict__ q;
        using pre_t = double2;
        __device__ __forceinline__ pre_t pre(int, size_t at) const
        {
            return ld2(p + at);
        }
        __device__ __forceinline__ double2 gather(int, size_t at) const
        {
            return ld2(p + at);
        }
        __device__ __forceinline__ double2 finish(size_t at, double2 s, const pre_t& pi) const
        {
            st2(q + at, s);
            return {pi.x * s.x, pi.y * s.y};
        }
    };

    // ------------------------------------------------------------ reductions
    __device__ __forceinline__ double2 blk_join(double2 a, double2 b, bool mx)
    {
        return mx ? double2{nanmax(a.x, b.x), nanmax(a.y, b.y)} : double2{a.x + b.x, a.y + b.y};
    }

    // The slots of s (slots x kl pairs, thread t's at t) joined in a tree; the result is
    // thread t's for t < kl.
    __device__ __forceinline__ double2 blk_fold(double2* s, int slots, int kl, bool mx)
    {
        const int t = threadIdx.x, w = t / kl;
        int       live = slots;
        while(live > 1)
        {
            const int half = (live + 1) / 2;
            __syncthreads();
            if(w + half < live)
                s[t] = blk_join(s[t], s[t + half * kl], mx);
            live = half;
        }
        return s[t];
    }

    // Per-column sum or maximum over the grid: thread t holds the pair t % kl.  The
    // CTA's partials go to red.partial, the last CTA adds them in a fixed order and
    // calls fin(column, value) once per column from one thread each.  The slots are
    // joined as a tree: with one pair 256 of them in a row cost 1.5 us twice a reduction
    // (2 columns on 40^2: 1.83 -> 1.58 ms a solve).
    template <class F>
    __device__ __forceinline__ void blk_reduce(double2 acc, int kl, bool mx, const blk_red& red,
                                               F&& fin)
    {
        __shared__ double2 s[kBlkNT];
        const int          t = threadIdx.x, slots = kBlkNT / kl, ld = 2 * kl;
        s[t] = acc;
        const double2 mine = blk_fold(s, slots, kl, mx);
        if(t < kl)
            st2(red.partial + (size_t)blockIdx.x * ld + 2 * t, mine);
        if(!grid_ticket(red.counter))
            return;
        double2 v{0.0, 0.0};
        if(t < slots * kl)
        {
            const double* p = red.partial + 2 * (t % kl);
#pragma unroll 4
            for(int b = t / kl; b < (int)gridDim.x; b += slots)
                v = blk_join(v, __ldcg(reinterpret_cast<const double2*>(p + (size_t)b * ld)), mx);
        }
        s[t] = v;
        v    = blk_fold(s, slots, kl, mx);
        if(t < kl)
        {
            fin(2 * t, v.x);
            fin(2 * t + 1, v.y);
        }
        if(t == 0)
            *red.counter = 0;
    }

    // ------------------------------------------------------------ row kernel
    // Threads of a CTA: (row slot, part of the row, column pair), the pair fastest.
    // Four CTAs per SM, one wave: at the 80 registers that the compiler takes without a
    // bound only three fit, and a grid of four per SM ran a second wave a third full
    // (32 right-hand sides on 64^3: 28.6 -> 25.1 ms; consecutive rows per CTA instead
    // of a grid stride: 25.6).
    // The next entries' columns and values are loaded while the gathers of the
    // current ones are in flight.
    template <class Op, class IT>
    __global__ void __launch_bounds__(kBlkNT, 4)
        k_blk_rows(csr_view<double, IT> A, Op op, int kl, int W, blk_red red)
    {
        constexpr int U = 4;
        if(red.skip && *red.skip)
            return;
        __shared__ double2 part[kBlkNT];
        const int          per  = kBlkNT / (kl * W); // rows of a CTA pass
        const int          pair = (int)threadIdx.x % kl;
        const int          w    = ((int)threadIdx.x / kl) % W;
        const int          slot = (int)threadIdx.x / (kl * W);
        const size_t       ld   = 2 * (size_t)kl;
        double2            acc{0.0, 0.0};
        for(int64_t base = (int64_t)blockIdx.x * per; base < A.m; base += (int64_t)gridDim.x * per)
        {
            const bool         valid = slot < per && base + slot < A.m;
            const int          row   = valid ? (int)(base + slot) : 0;
            const size_t       at    = (size_t)row * ld + 2 * pair;
            double2            s{0.0, 0.0};
            typename Op::pre_t pr{};
            if(valid)
            {
                const int b = A.rp[row + 1];
                int       j = A.rp[row] + w;
                if(w == 0)
                    pr = op.pre(row, at);
                double v[U];
                int    c[U];
#pragma unroll
                for(int u = 0; u < U; u++)
                    if(j + u * W < b)
                    {
                        v[u] = __ldg(A.v + j + u * W);
                        c[u] = col_of<IT>(__ldg(A.ci + j + u * W), row);
                    }
#pragma unroll 1
                for(; j < b; j += U * W)
                {
                    double2 g[U];
                    double  vn[U];
                    int     cn[U];
#pragma unroll
                    for(int u = 0; u < U; u++)
                        if(j + u * W < b)
                            g[u] = op.gather(c[u], (size_t)c[u] * ld + 2 * pair);
#pragma unroll
                    for(int u = 0; u < U; u++)
                        if(j + (U + u) * W < b)
                        {
                            vn[u] = __ldg(A.v + j + (U + u) * W);
                            cn[u] = col_of<IT>(__ldg(A.ci + j + (U + u) * W), row);
                        }
#pragma unroll
                    for(int u = 0; u < U; u++)
                        if(j + u * W < b)
                        {
                            s.x = fma(v[u], g[u].x, s.x);
                            s.y = fma(v[u], g[u].y, s.y);
                        }
#pragma unroll
                    for(int u = 0; u < U; u++)
                    {
                        v[u] = vn[u];
                        c[u] = cn[u];
                    }
                }
            }
            if(W > 1)
            {
                part[threadIdx.x] = s;
                __syncthreads();
                if(valid && w == 0)
                    for(int q = 1; q < W; q++)
                        s = blk_join(s, part[threadIdx.x + q * kl], false);
                __syncthreads();
            }
            if(valid && w == 0)
            {
                const double2 d = op.finish(at, s, pr);
                if(Op::kDot)
                {
                    acc.x += d.x;
                    acc.y += d.y;
                }
            }
        }
        if(Op::kDot)
            blk_reduce(acc, kl, false, red,
                       [&](int c, double v) { red.out[(size_t)c * red.stride] = v; });
    }

    // W: interleaved parts of a row.  Below about 1024 threads per SM the pass waits on
    // the row -> entries -> gathers chain, so rows are split until the grid reaches
    // that or a part is down to four entries.
    template <class Op>
    static lab_status blk_rows(const lab_csr_impl* A, const Op& op, int ld, cudaStream_t s,
                               const blk_red& red)
    {
        if(A->m == 0)
            return LAB_OK;
        const int kl = ld / 2;
        int       W  = 1;
        while(W < 16 && 2 * W * kl <= kBlkNT && A->m * kl * W < (int64_t)num_sms() * 1024 &&
              A->nnz >= 8 * A->m * W)
            W *= 2;
        const int64_t  per  = kBlkNT / (kl * W);
        const unsigned grid =
            (unsigned)std::min<int64_t>(ceil_div<int64_t>(A->m, per), kBlkRedGrid);
        if(A->lp.dcol)
        {
            csr_view<double, int16_t> V{A->row_ptr, A->lp.dcol, A->val, (int32_t)A->m};
            LAB_LAUNCH((k_blk_rows<Op, int16_t>), grid, kBlkNT, 0, s, V, op, kl, W, red);
        }
        else
        {
            csr_view<double, int32_t> V{A->row_ptr, A->col_ind, A->val, (int32_t)A->m};
            LAB_LAUNCH((k_blk_rows<Op, int32_t>), grid, kBlkNT, 0, s, V, op, kl, W, red);
        }
        return LAB_OK;
    }

    // ------------------------------------------------------------ layout
    // Column-major columns to interleaved and back, 32 rows by up to 32 columns through
    // shared memory so both sides are coalesced.
    __global__ void k_to_blk(const double* __restrict__ x, int64_t ldx, int64_t n, int ncols,
                             int ld, double* __restrict__ xb)
    {
        __shared__ double t[32][33];
        const int64_t     i0 = (int64_t)blockIdx.x * 32;
        for(int c0 = 0; c0 < ld; c0 += 32)
        {
            for(int c = c0 + threadIdx.y; c < min(c0 + 32, ld); c += blockDim.y)
                t[c - c0][threadIdx.x] =
                    c < ncols && i0 + threadIdx.x < n ? x[c * ldx + i0 + threadIdx.x] : 0.0;
            __syncthreads();
            for(int r = threadIdx.y; r < 32; r += blockDim.y)
                if(i0 + r < n && c0 + (int)threadIdx.x < ld)
                    xb[(i0 + r) * ld + c0 + threadIdx.x] = t[threadIdx.x][r];
            __syncthreads();
        }
    }

    __global__ void k_from_blk(const double* __restrict__ xb, int64_t n, int ncols, int ld,
                               double* __restrict__ x, int64_t ldx)
    {
        __shared__ double t[32][33];
        const int64_t     i0 = (int64_t)blockIdx.x * 32;
        for(int c0 = 0; c0 < ncols; c0 += 32)
        {
            for(int r = threadIdx.y; r < 32; r += blockDim.y)
                if(i0 + r < n && c0 + (int)threadIdx.x < ncols)
                    t[r][threadIdx.x] = xb[(i0 + r) * ld + c0 + threadIdx.x];
            __syncthreads();
            for(int c = c0 + threadIdx.y; c < min(c0 + 32, ncols); c += blockDim.y)
                if(i0 + threadIdx.x < n)
                    x[c * ldx + i0 + threadIdx.x] = t[threadIdx.x][c - c0];
            __syncthreads();
        }
    }

    lab_status blk_from_columns(const double* x, int64_t ldx, int64_t n, int ncols, int ld,
                                double* xb, cudaStream_t s)
    {
        LAB_LAUNCH(k_to_blk, (unsigned)ceil_div<int64_t>(n, 32), dim3(32, 8), 0, s, x, ldx, n, ncols,
                   ld, xb);
        return LAB_OK;
    }

    lab_status blk_to_columns(const double* xb, int64_t n, int ncols, int ld, double* x,
                              int64_t ldx, cudaStream_t s)
    {
        LAB_LAUNCH(k_from_blk, (unsigned)ceil_div<int64_t>(n, 32), dim3(32, 8), 0, s, xb, n, ncols,
                   ld, x, ldx);
        return LAB_OK;
    }

    // ------------------------------------------------------------ PCG vector passes
    __device__ __forceinline__ void blk_retire(int* sf, int c, int* gflags, int status, int conv)
    {
        sf[c * GF_N + GF_DONE]   = 1;
        sf[c * GF_N + GF_CONV]   = conv;
        sf[c * GF_N + GF_STATUS] = status;
        if(atomicSub(&gflags[1], 1) == 1)
            gflags[0] = 1;
    }

    // ||r||_inf per column into sc[c][G_R0]
    __global__ void __launch_bounds__(kBlkNT)
        k_blk_norm(int64_t n, int kl, const double* __restrict__ r, blk_red red)
    {
        const int    pair = (int)threadIdx.x % kl, slot = (int)threadIdx.x / kl;
        const int    per  = kBlkNT / kl;
        double2      acc{0.0, 0.0};
        if(slot < per)
            for(int64_t i = (int64_t)blockIdx.x * per + slot; i < n; i += (int64_t)gridDim.x * per)
            {
                const double2 v = ld2(r + i * 2 * kl + 2 * pair);
                acc             = blk_join(acc, {fabs(v.x), fabs(v.y)}, true);
            }
        blk_reduce(acc, kl, true, red,
                   [&](int c, double v) { red.out[(size_t)c * red.stride] = v; });
    }

    // gamma = (z, r), p = z is set by the caller; columns with r = 0 retire at once.
    __global__ void k_blk_init(double* sc, int* sf, int* gflags, int ld, int max_iter)
    {
        int active = 0;
        for(int c = threadIdx.x; c < ld; c += 32)
        {
            sc[c * G_N + G_GAMMA]    = sc[c * G_N + G_GNEW];
            sc[c * G_N + G_RN]       = sc[c * G_N + G_R0];
            const bool zero          = sc[c * G_N + G_R0] == 0.0;
            sf[c * GF_N + GF_ITER]   = 0;
            sf[c * GF_N + GF_DONE]   = zero;
            sf[c * GF_N + GF_CONV]   = zero;
            sf[c * GF_N + GF_STATUS] = zero ? LAB_OK : LAB_NOT_CONVERGED;
            active += !zero;
        }
        for(int o = 16; o > 0; o >>= 1)
            active += __shfl_xor_sync(0xffffffffu, active, o);
        if(threadIdx.x == 0)
        {
            gflags[1] = active;
            gflags[2] = max_iter;
            gflags[0] = active == 0;
        }
    }

    // x += alpha p; r -= alpha q; ||r||_inf; stopping test, per column (k_seg_update)
    __global__ void __launch_bounds__(kBlkNT)
        k_blk_update(int64_t n, int kl, double* __restrict__ x, double* __restrict__ r,
                     const double* __restrict__ p, const double* __restrict__ q, double* sc, int* sf,
                     int* gflags, blk_red red, double rtol, double atol)
    {
        if(gflags[0])
            return;
        const int    pair = (int)threadIdx.x % kl, slot = (int)threadIdx.x / kl;
        const int    per  = kBlkNT / kl;
        const int    c0   = 2 * pair;
        const bool   d0 = sf[c0 * GF_N + GF_DONE], d1 = sf[(c0 + 1) * GF_N + GF_DONE];
        const double a0 = sc[c0 * G_N + G_GAMMA] / sc[c0 * G_N + G_PQ];
        const double a1 = sc[(c0 + 1) * G_N + G_GAMMA] / sc[(c0 + 1) * G_N + G_PQ];
        double2      acc{0.0, 0.0};
        if(slot < per && !(d0 && d1))
        {
#pragma unroll 2
            for(int64_t i = (int64_t)blockIdx.x * per + slot; i < n; i += (int64_t)gridDim.x * per)
            {
                const size_t  at = (size_t)i * 2 * kl + c0;
                const double2 pv = ld2(p + at), qv = ld2(q + at);
                double2       xv = *reinterpret_cast<const double2*>(x + at);
                double2       rv = *reinterpret_cast<const double2*>(r + at);
                if(!d0)
                {
                    xv.x = __dadd_rn(__dmul_rn(a0, pv.x), xv.x);
                    rv.x = __dadd_rn(__dmul_rn(-a0, qv.x), rv.x);
                }
                if(!d1)
                {
                    xv.y = __dadd_rn(__dmul_rn(a1, pv.y), xv.y);
                    rv.y = __dadd_rn(__dmul_rn(-a1, qv.y), rv.y);
                }
                st2(x + at, xv);
                st2(r + at, rv);
                acc = blk_join(acc, {fabs(rv.x), fabs(rv.y)}, true);
            }
        }
        blk_reduce(acc, kl, true, red, [&](int c, double t) {
            if(sf[c * GF_N + GF_DONE])
                return;
            sc[c * G_N + G_RN] = t;
            const double r0    = sc[c * G_N + G_R0];
            const bool   nan   = isnan(t) || isnan(r0);
            if(!nan && (t <= atol || t / r0 <= rtol))
                blk_retire(sf, c, gflags, LAB_OK, 1);
            else if(nan)
                blk_retire(sf, c, gflags, LAB_NAN, 0);
        });
    }

    // p = z + beta p, then (last CTA) gamma <- gnew, iteration count, max_iter test
    __global__ void __launch_bounds__(kBlkNT)
        k_blk_pupdate(int64_t n, int kl, double* __restrict__ p, const double* __restrict__ z,
                      double* sc, int* sf, int* gflags, unsigned int* counter)
    {
        if(gflags[0])
            return;
        const int    pair = (int)threadIdx.x % kl, slot = (int)threadIdx.x / kl;
        const int    per  = kBlkNT / kl;
        const int    c0   = 2 * pair;
        const bool   d0 = sf[c0 * GF_N + GF_DONE], d1 = sf[(c0 + 1) * GF_N + GF_DONE];
        const double b0 = sc[c0 * G_N + G_GNEW] / sc[c0 * G_N + G_GAMMA];
        const double b1 = sc[(c0 + 1) * G_N + G_GNEW] / sc[(c0 + 1) * G_N + G_GAMMA];
        if(slot < per && !(d0 && d1))
        {
#pragma unroll 4
            for(int64_t i = (int64_t)blockIdx.x * per + slot; i < n; i += (int64_t)gridDim.x * per)
            {
                const size_t  at = (size_t)i * 2 * kl + c0;
                const double2 zv = ld2(z + at);
                double2       pv = *reinterpret_cast<const double2*>(p + at);
                if(!d0)
                    pv.x = b0 == 0.0 ? zv.x : __dadd_rn(zv.x, __dmul_rn(b0, pv.x));
                if(!d1)
                    pv.y = b1 == 0.0 ? zv.y : __dadd_rn(zv.y, __dmul_rn(b1, pv.y));
                st2(p + at, pv);
            }
        }
        if(!grid_ticket(counter))
            return;
        for(int c = threadIdx.x; c < 2 * kl; c += kBlkNT)
            if(!sf[c * GF_N + GF_DONE])
            {
                sc[c * G_N + G_GAMMA]  = sc[c * G_N + G_GNEW];
                const int it           = sf[c * GF_N + GF_ITER] + 1;
                sf[c * GF_N + GF_ITER] = it;
                if(it > gflags[2])
                    blk_retire(sf, c, gflags, LAB_NOT_CONVERGED, 0);
            }
        if(threadIdx.x == 0)
            *counter = 0;
    }

    static unsigned blk_grid(int64_t n, int kl)
    {
        return (unsigned)std::max<int64_t>(
            1, std::min<int64_t>(ceil_div<int64_t>(n, kBlkNT / kl), kBlkRedGrid));
    }

    lab_status blk_norm(int64_t n, int ld, const double* r, const blk_red& red, cudaStream_t s)
    {
        LAB_LAUNCH(k_blk_norm, blk_grid(n, ld / 2), kBlkNT, 0, s, n, ld / 2, r, red);
        return LAB_OK;
    }
    lab_status blk_init(double* sc, int* sf, int* gflags, int ld, int max_iter, cudaStream_t s)
    {
        LAB_LAUNCH(k_blk_init, 1, 32, 0, s, sc, sf, gflags, ld, max_iter);
        return LAB_OK;
    }
    lab_status blk_update(int64_t n, int ld, double* x, double* r, const double* p, const double* q,
                          double* sc, int* sf, int* gflags, const blk_red& red, double rtol,
                          double atol, cudaStream_t s)
    {
        LAB_LAUNCH(k_blk_update, blk_grid(n, ld / 2), kBlkNT, 0, s, n, ld / 2, x, r, p, q, sc, sf,
                   gflags, red, rtol, atol);
        return LAB_OK;
    }
    lab_status blk_pupdate(int64_t n, int ld, double* p, const double* z, double* sc, int* sf,
                           int* gflags, unsigned int* counter, cudaStream_t s)
    {
        LAB_LAUNCH(k_blk_pupdate, blk_grid(n, ld / 2), kBlkNT, 0, s, n, ld / 2, p, z, sc, sf,
                   gflags, counter);
        return LAB_OK;
    }
    lab_status blk_spmv_dot(const lab_csr_impl* A, int ld, const double* p, double* q,
                            const blk_red& red, cudaStream_t s)
    {
        return blk_rows(A, bop_spmv_dot{p, q}, ld, s, red);
    }
    lab_status blk_residual(const lab_csr_impl* A, int ld, const double* x, const double* b,
                            double* r, cudaStream_t s)
    {
        return blk_rows(A, bop_res{x, b, r}, ld, s, blk_red{});
    }

    // ------------------------------------------------------------ small kernels
    __global__ void k_blk_zero(double* x, int64_t n, const int* skip)
    {
        if(skip && *skip)
            return;
        for(int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
            i += (int64_t)gridDim.x * blockDim.x)
            x[i] = 0.0;
    }

    // Coarsest level per column: x = b / a (1x1).
    __global__ void k_blk_coarse1(const double* __restrict__ a, const double* __restrict__ b,
                                  double* __restrict__ x, int ld, const int* skip)
    {
        if(skip && *skip)
            return;
        const int c = threadIdx.x;
        if(c < ld)
            x[c] = __ddiv_rn(b[c], a[0]);
    }

    // Coarsest level, dense inverse: x = Ainv b.  A CTA has R rows; its threads are (part
    // of the row, column pair), the pair fastest, so a warp reads neighbouring entries
    // of b's rows and a run of Ainv's row (one entry a warp with 64 columns), and an
    // entry of b serves R rows.  The parts, interleaved, are added as a tree.  A solve of 2
    // / 32 columns with 1171 coarsest rows takes 1.6 / 3.5 ms, with 4031 rows 1.8 / 5.8 ms
    // (a thread per row and column that sums its row alone, waiting for that chain: 4.4 /
    // 6.5 and 26.4 / 16.1 ms).
    template <int R>
    __global__ void __launch_bounds__(kBlkNT)
        k_blk_dense(const double* __restrict__ a, const double* __restrict__ b,
                    double* __restrict__ x, int n, int kl, const int* skip)
    {
        if(skip && *skip)
            return;
        __shared__ double2 part[R][kBlkNT];
        const int          t = threadIdx.x, parts = kBlkNT / kl, pair = t % kl, w = t / kl;
        const int          row = (int)blockIdx.x * R, ld = 2 * kl;
        double2            s[R];
#pragma unroll
        for(int r = 0; r < R; r++)
            s[r] = {0.0, 0.0};
        if(w < parts)
        {
#pragma unroll 4
            for(int j = w; j < n; j += parts)
            {
                const double2 v = ld2(b + (size_t)j * ld + 2 * pair);
#pragma unroll
                for(int r = 0; r < R; r++)
                {
                    // rows past the last one read it again
                    const double e = __ldg(a + (size_t)min(row + r, n - 1) * n + j);
                    s[r].x         = fma(e, v.x, s[r].x);
                    s[r].y         = fma(e, v.y, s[r].y);
                }
            }
        }
#pragma unroll
        for(int r = 0; r < R; r++)
            part[r][t] = s[r];
        int live = parts;
        while(live > 1)
        {
            const int half = (live + 1) / 2;
            __syncthreads();
            if(w + half < live)
#pragma unroll
                for(int r = 0; r < R; r++)
                    part[r][t] = blk_join(part[r][t], part[r][t + half * kl], false);
            live = half;
        }
        if(t < kl)
#pragma unroll
            for(int r = 0; r < R; r++)
                if(row + r < n)
                    st2(x + (size_t)(row + r) * ld + 2 * t, part[r][t]);
    }

    // (z, r) where the cycle's last pass does not form it
    __global__ void __launch_bounds__(kBlkNT)
        k_blk_dot(int64_t n, int kl, const double* __restrict__ x, const double* __restrict__ y,
                  blk_red red)
    {
        if(red.skip && *red.skip)
            return;
        const int    pair = (int)threadIdx.x % kl, slot = (int)threadIdx.x / kl;
        const int    per  = kBlkNT / kl;
        double2      acc{0.0, 0.0};
        if(slot < per)
            for(int64_t i = (int64_t)blockIdx.x * per + slot; i < n; i += (int64_t)gridDim.x * per)
            {
                const double2 u = ld2(x + i * 2 * kl + 2 * pair), v = ld2(y + i * 2 * kl + 2 * pair);
                acc.x += u.x * v.x;
                acc.y += u.y * v.y;
            }
        blk_reduce(acc, kl, false, red,
                   [&](int c, double v) { red.out[(size_t)c * red.stride] = v; });
    }

    // ------------------------------------------------------------ the recursion
    // x = cycle(0; b) on level l; x0_ready: the restriction wrote the first sweep into
    // the buffer that the cycle starts in; dot (level 0): (x, b) per column.
    static bool blk_starts_in_t(const lab_amg_options* o)
    {
        // start in the buffer that makes the last write land in x
        return (((o->n1 >= 1 ? o->n1 - 1 : o->n1) + 1 + o->n2) & 1) != 0;
    }

    static lab_status cycle_blk(hierarchy_impl* h, int l, int ld, double* x, const double* b,
                                const cyc_ctx& c, bool x0_ready, const blk_red& dot)
    {
        const lab_amg_options* o = c.o;
        lab_csr_impl*          A = h->A[l];
        const int64_t          m = A->m;
        blk_red                none{};
        none.skip = c.skip;
        auto dotted = [&]() -> lab_status {
            if(dot.out)
                LAB_LAUNCH(k_blk_dot, blk_grid(m, ld / 2), kBlkNT, 0, c.s, m, ld / 2,
                           (const double*)x, b, dot);
            return LAB_OK;
        };
        if(l == h->levels)
        {
            const double* inv = h->coarse_inv;
            if(m == 1)
                LAB_LAUNCH(k_blk_coarse1, 1, kBlkMax, 0, c.s, (const double*)A->val, b, x, ld,
                           c.skip);
            else if(m > 4 * num_sms()) // a row per CTA fills the GPU up to there
                LAB_LAUNCH(k_blk_dense<4>, (unsigned)ceil_div<int64_t>(m, 4), kBlkNT, 0, c.s, inv, b,
                           x, (int)m, ld / 2, c.skip);
            else if(m > 1)
                LAB_LAUNCH(k_blk_dense<1>, (unsigned)m, kBlkNT, 0, c.s, inv, b, x, (int)m, ld / 2,
                           c.skip);
            return dotted();
        }
        lab_csr_impl* P    = h->P[l];
        lab_csr_impl* R    = h->R[l];
        level_ws&     w    = h->ws[l];
        level_ws&     wc   = h->ws[l + 1];
        const int     n1   = o->n1, n2 = o->n2;
        const double  om   = o->omega;
        const double* invd = A->invdiag;
        double*       r    = w.rk;
        double*       cur  = x;
        double*       oth  = w.tk;
        if(blk_starts_in_t(o))
            std::swap(cur, oth);
        auto jacobi = [&](bool last) -> lab_status {
            if(last && dot.out)
                LAB_TRY(blk_rows(A, bop_jacobi<true>{cur, b, invd, om, oth}, ld, c.s, dot));
            else
                LAB_TRY(blk_rows(A, bop_jacobi<false>{cur, b, invd, om, oth}, ld, c.s, none));
            std::swap(cur, oth);
            return LAB_OK;
        };
        if(n1 >= 1)
        {
            if(x0_ready)
                LAB_TRY(blk_rows(A, bop_res{cur, b, r}, ld, c.s, none));
            else
                LAB_TRY(blk_rows(A, bop_pre0{b, invd, om, cur, r}, ld, c.s, none));
            for(int k = 1; k < n1; k++)
                LAB_TRY(jacobi(false));
            if(n1 > 1)
                LAB_TRY(blk_rows(A, bop_res{cur, b, r}, ld, c.s, none));
        }
        else
        {
            LAB_LAUNCH(k_blk_zero, grid_for(m * ld), 256, 0, c.s, cur, m * ld, c.skip);
            LAB_TRY(blk_rows(A, bop_res{cur, b, r}, ld, c.s, none));
        }
        const bool fuse = n1 >= 1 && l + 1 < h->levels;
        double*    x0   = fuse ? (blk_starts_in_t(o) ? wc.tk : wc.xk) : nullptr;
        LAB_TRY(blk_rows(R, bop_restrict{r, wc.bk, h->A[l + 1]->invdiag, om, x0}, ld, c.s, none));
        LAB_TRY(cycle_blk(h, l + 1, ld, wc.xk, wc.bk, c, fuse, blk_red{}));
        LAB_TRY(blk_rows(P, bop_prolong{wc.xk, cur, oth}, ld, c.s, none));
        std::swap(cur, oth);
        for(int k = 0; k < n2; k++)
            LAB_TRY(jacobi(k == n2 - 1));
        if(cur != x)
        {
            set_error("block cycle: internal buffer parity");
            return LAB_BAD_ARG;
        }
        return n2 > 0 ? LAB_OK : dotted();
    }

    bool cycle_block_supported(const hierarchy_impl* h, const lab_amg_options* o)
    {
        if(o->cycle != LAB_CYCLE_V || o->smoother != LAB_SMOOTH_JACOBI ||
           o->precision != LAB_PREC_FP64 || o->n1 < 0 || o->n2 < 0 || h->A[0]->m == 0)
            return false;
        const lab_csr_impl* Ac = h->A[h->levels];
        return Ac->m <= 1 || (o->coarse == LAB_COARSE_DIRECT && h->coarse_inv);
    }

    lab_status cycle_prepare_block(hierarchy_impl* h, int ld, int vectors, cudaStream_t s)
    {
        int64_t rows = (int64_t)(vectors + 2) * h->A[0]->m;
        for(int l = 1; l <= h->levels; l++)
            rows += 4 * h->A[l]->m;
        const int64_t bytes = rows * ld * (int64_t)sizeof(double);
        if(h->block_bytes && bytes > h->block_bytes)
        {
            set_error("a block of %d columns needs %lld bytes", ld, (long long)bytes);
            return LAB_OOM;
        }
        for(int l = 0; l <= h->levels; l++)
        {
            level_ws& w = h->ws[l];
            if(w.kcols >= ld)
                continue;
            double** v[4] = {&w.xk, &w.bk, &w.rk, &w.tk};
            w.kcols       = 0;
            for(double** p : v)
            {
                dfree(*p, s);
                *p = nullptr;
                // level 0 works on the solve's own vectors and needs scratch alone
                if(l > 0 || p == &w.rk || p == &w.tk)
                    LAB_TRY(dalloc(p, (size_t)h->A[l]->m * ld + 2, s));
            }
            w.kcols = ld;
        }
        return LAB_OK;
    }

    // A workspace of up to 64 MB, or of 256 bytes a row of the hierarchy (four vectors of
    // eight columns), stays for the next solve; allocating a larger one again, from the
    // pool, does not show (32 columns on 64^3: 23.8 ms either way).
    void cycle_release_block(hierarchy_impl* h, bool if_large, cudaStream_t s)
    {
        int64_t rows = 0, held = 0;
        for(int l = 0; l <= h->levels; l++)
        {
            rows += h->A[l]->m;
            held += (l ? 4 : 2) * h->A[l]->m * h->ws[l].kcols * (int64_t)sizeof(double);
        }
        if(if_large && held <= std::max<int64_t>(256 * rows, 64 << 20))
            return;
        for(int l = 0; l <= h->levels; l++)
        {
            level_ws& w = h->ws[l];
            for(double** p : {&w.xk, &w.bk, &w.rk, &w.tk})
            {
                dfree(*p, s);
                *p = nullptr;
            }
            w.kcols = 0;
        }
    }

    lab_status cycle_precond_block(hierarchy_impl* h, const cyc_ctx& c, int ld, const double* r,
                                   double* z, const blk_red& dot)
    {
        return cycle_blk(h, 0, ld, z, r, c, false, dot);
    }
}
