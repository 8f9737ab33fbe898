// The last levels of a V-cycle in one launch (see cycle.cu for the per-pass form).
#include "cycle.cuh"

namespace lab
{
    // ================================================================ fused tail
    // The last levels of a V-cycle with Jacobi smoothing from a zero guess hold a
    // few hundred rows each, so their passes (restriction, residual, smoothing,
    // prolongation, the coarsest solve) cost launch and round-trip latency, not
    // bandwidth.  One CTA runs them all, from the restriction out of the entry
    // level p to the prolongation back into it, passes separated by block
    // barriers.
    //
    // A pass that reads its operator from L2 waits three dependent round trips (row
    // bounds, entries, gathers) of 600 to 1400 cycles each.  So what the passes
    // touch lives in shared memory: the operators' row pointers, columns and values
    // (and the iterate of level p) arrive by bulk copies in flight while the
    // residual of level p is gathered, entry by entry over the whole CTA, to the
    // positions of R's entries; the level vectors never leave the SM.  The passes
    // are a list of descriptors with shared-memory offsets, made on the host and
    // copied to shared memory first (reading a few fields of a large kernel argument
    // in every pass cost 1000 cycles a pass), run by one loop; the warps without a
    // row go straight to the barrier.
    //
    // Measured (one launch a cycle; before, with operators and vectors in global
    // memory): 64^2 Poisson 34 -> 13 us and 1.35 -> 1.08 ms for the CG solve, 128^3
    // Poisson 41 -> 10 us, 80^3 graph Laplacian 48 -> 6 us plus two launches, 8.9 -> 8.0
    // ms for the adjoint solve.  Bound by the chain of shared-memory latencies, 850 to
    // 1000 cycles for the smallest pass.
    //
    // Each row is summed in its operator's schedule order (CSR order for the
    // one-thread-per-row plan, k_vector's lane order and xor tree for W lanes), with
    // the ops' own epilogue arithmetic, so the result equals the per-pass launches
    // bit for bit.
    constexpr int    kTailMax    = 8;
    constexpr int    kTailNT     = 512;
    constexpr int    kTailEdge   = 4096; // entries of R and P that the launch takes in
    constexpr int    kTailPasses = 48;
    constexpr int    kTailCopies = 96;
    constexpr size_t kTailSmem   = 216 * 1024; // operators and vectors of one launch

    // What a pass does with a row's sum s.
    enum
    {
        TAIL_RES,      // y_i = b_i - s
        TAIL_JACOBI,   // y_i = x_i + omega (D^-1_i (b_i - s))
        TAIL_RESTRICT, // y_i = s; z_i = omega (D^-1_i s)
        TAIL_PROLONG,  // y_i = x_i + s
        TAIL_SCALE,    // z_i = omega (D^-1_i b_i), no operator
        TAIL_COARSE    // y = b / a (1x1) or Ainv b, no operator
    };
    // Where a pass reads its columns: absolute, relative to the row, or x already
    // gathered to the positions of the entries.
    enum
    {
        TAIL_COL,
        TAIL_DCOL,
        TAIL_GATHERED
    };
    // Read as four 16-byte words.  Offsets are bytes in shared memory; those of
    // vectors that the pass does not use are 0 (read, not used), y and z -1 when not
    // written there.
    struct alignas(16) tail_pass
    {
        int m, lw;           // rows; log2 of the lanes per row (0: CSR order)
        int mode, cols;
        int o_rp, o_ci, o_v; // the operator
        int out;             // y goes to the launch's result
        int in, y, x, b;
        int invd, z, pad[2];
    };
    struct tail_copy
    {
        const void* src;
        int         off, bytes;
    };
    struct tail_args
    {
        tail_pass     pass[kTailPasses];
        tail_copy     copy[kTailCopies];
        int           npass, ncopy, bytes; // bytes: of all copies
        // the first pass's gather: xg[j] = wr[ci[j]], j < gnnz <= kTailEdge
        const int32_t* gci;
        const void*    wr;
        int            gnnz, gx;
        double         omega;
        const double*  a11;  // coarsest 1x1: its value
        const double*  ainv; // coarsest n x n: dense inverse (o_v of its pass: local copy)
        int            nc;
        void*          dst; // the launch's result
        int            ndst;
        const int*     skip;
        // counts of waits that ran out (the device's, the hierarchy's), the bound in
        // polls, and 1 for an arrival that never comes (the test of the bound)
        int *          status, *timeouts;
        unsigned       polls;
        int            held;
    };

    template <class T, class IT>
    __device__ __forceinline__ T tail_x(const T* x, const IT* ci, int j, int row)
    {
        if constexpr(std::is_void<IT>::value)
            return x[j];
        else
            return x[col_of<IT>(ci[j], row)];
    }

    // The rows of one pass.  A pass is a chain of shared-memory latencies, so what
    // does not depend on one another is loaded together and without branches
    // (positions outside the row at a clamped one inside it, the sum unchanged).  A
    // row without entries, and a lane past the last row, has no position inside it
    // and loads none: its loop starts at its end (the quad below starts before
    // the row, so it would be entered, and what lies past the operator's last entry
    // is no column).
    template <class T, class IT>
    __device__ __forceinline__ void tail_rows(const int4 q0, const int4 q1, const int4 q2,
                                              const int4 q3, unsigned char* sm, T om, T* dst)
    {
        constexpr int  U    = 4;
        const int      m = q0.x, lw = q0.y, mode = q0.z;
        const int      W = 1 << lw, per = kTailNT >> lw;
        const int      lane = (int)threadIdx.x & (W - 1);
        const int32_t* rp   = reinterpret_cast<const int32_t*>(sm + q1.x);
        const IT*      ci   = reinterpret_cast<const IT*>(sm + q1.y);
        const T*       v    = reinterpret_cast<const T*>(sm + q1.z);
        const T*       in   = reinterpret_cast<const T*>(sm + q2.x);
        // FP64 and CSR order: entries lane, lane + W, ...; reduced precision with W
        // lanes: k_vector's aligned quads
        const bool quad = sizeof(T) == 4 && W > 1;
        const int  st   = quad ? 1 : W;
#pragma unroll 1
        for(int row = (int)threadIdx.x >> lw; row - (((int)threadIdx.x & 31) >> lw) < m; row += per)
        {
            const int r  = min(row, m - 1);
            const int a0 = rp[r], a1 = row < m ? rp[r + 1] : a0;
            const T   px = reinterpret_cast<const T*>(sm + q2.z)[r];
            const T   pb = reinterpret_cast<const T*>(sm + q2.w)[r];
            const T   pd = reinterpret_cast<const T*>(sm + q3.x)[r];
            T         s  = T(0);
#pragma unroll 1
            for(int j = a0 == a1 ? a1 : quad ? (a0 & ~3) + 4 * lane : a0 + lane; j < a1;
                j += U * W)
            {
                T vv[U], xv[U];
#pragma unroll
                for(int u = 0; u < U; u++)
                {
                    const int k = max(a0, min(j + u * st, a1 - 1));
                    vv[u]       = v[k];
                    xv[u]       = tail_x<T, IT>(in, ci, k, row);
                }
#pragma unroll
                for(int u = 0; u < U; u++)
                {
                    const T t = acc_step<true>(vv[u], xv[u], s);
                    s         = j + u * st >= a0 && j + u * st < a1 ? t : s;
                }
            }
#pragma unroll 1
            for(int o = W >> 1; o > 0; o >>= 1)
                s += __shfl_xor_sync(0xffffffffu, s, o, W);
            if(row < m && lane == 0)
            {
                const T res = pb - s;
                T       yi  = mode == TAIL_RES ? res : s;
                if(mode == TAIL_JACOBI)
                    yi = px + om * (pd * res);
                if(mode == TAIL_PROLONG)
                    yi = px + s;
                if(q1.w)
                    dst[row] = yi;
                else
                    reinterpret_cast<T*>(sm + q2.y)[row] = yi;
                if(q3.y >= 0)
                    reinterpret_cast<T*>(sm + q3.y)[row] = om * (pd * s);
            }
        }
    }

    template <class T>
    __global__ void __launch_bounds__(kTailNT, 1) k_tail(const __grid_constant__ tail_args a)
    {
        extern __shared__ __align__(128) unsigned char smem_tail[];
        __shared__ __align__(16) tail_pass  s_pass[kTailPasses];
        __shared__ __align__(8) uint64_t    bar;
        unsigned char*                      sm = smem_tail;
        // read now, looked at after the gather: a skipped launch writes nothing
        const int     skip = a.skip ? __ldcg(a.skip) : 0;
        const double  a11  = a.nc == 1 ? __ldg(a.a11) : 0.0;
        const int     warp = threadIdx.x >> 5;
        constexpr int G    = kTailEdge / kTailNT;
        int           gc[G];
#pragma unroll
        for(int u = 0; u < G; u++)
        {
            const int j = (int)threadIdx.x + u * kTailNT;
            gc[u]       = j < a.gnnz ? __ldg(a.gci + j) : -1;
        }
        if(threadIdx.x == 0)
        {
            mbar_init(&bar, 1 + a.held);
            fence_barrier_init();
            mbar_arrive_expect_tx(&bar, (unsigned)a.bytes);
        }
        __syncthreads();
        // a warp per copy and per descriptor: one read of the argument at a uniform
        // address each
        if((threadIdx.x & 31) == 0)
        {
#pragma unroll 1
            for(int i = warp; i < a.ncopy; i += kTailNT / 32)
                bulk_g2s(sm + a.copy[i].off, a.copy[i].src, (unsigned)a.copy[i].bytes, &bar);
#pragma unroll 1
            for(int i = warp; i < a.npass; i += kTailNT / 32)
                s_pass[i] = a.pass[i];
        }
        const T om = (T)a.omega;
        {
            // the residual at each entry's column of the first pass
            const T* wr = static_cast<const T*>(a.wr);
            T*       xg = reinterpret_cast<T*>(sm + a.gx);
            T        g[G];
#pragma unroll
            for(int u = 0; u < G; u++)
                if(gc[u] >= 0)
                    g[u] = __ldg(wr + gc[u]);
#pragma unroll
            for(int u = 0; u < G; u++)
                if(gc[u] >= 0)
                    xg[threadIdx.x + u * kTailNT] = g[u];
        }
        // every copy has landed; a wait that runs out makes the result NaN (no solve goes
        // on with it), counts itself, drains (bounded) and leaves
        {
            bool ok = false;
            for(unsigned i = 0; i < a.polls && !ok; i++)
                ok = mbar_try_wait(&bar, 0);
            if(__syncthreads_or(!ok))
            {
                if(!skip)
                    for(int i = threadIdx.x; i < a.ndst; i += kTailNT)
                        static_cast<T*>(a.dst)[i] = (T)__longlong_as_double(0x7ff8000000000000ll);
                if(threadIdx.x == 0)
                {
                    atomicAdd(a.status, 1);
                    atomicAdd(a.timeouts, 1);
                    if(a.held)
                        mbar_arrive(&bar);
                    for(unsigned i = 0; i < kStreamWaitLimit && !mbar_try_wait(&bar, 0); i++)
                        ;
                }
                return;
            }
        }
        if(skip)
            return;
        const int npass = a.npass;
        T*        dst   = static_cast<T*>(a.dst);
#pragma unroll 1
        for(int p = 0; p < npass; p++)
        {
            const int4* q  = reinterpret_cast<const int4*>(s_pass + p);
            const int4  q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];
            // the warps beyond the last row go straight to the barrier
            if((warp << 5) >> q0.y < q0.x)
            {
                if(q0.z == TAIL_COARSE)
                {
                    // coarsest level: x = b / a (1x1) or x = Ainv b (k_coarse1,
                    // k_coarse_dense)
                    const T* b = reinterpret_cast<const T*>(sm + q2.w);
                    T*       x = q1.w ? dst : reinterpret_cast<T*>(sm + q2.y);
                    if(a.nc == 1)
                    {
                        if(threadIdx.x == 0)
                            x[0] = (T)__ddiv_rn((double)b[0], a11);
                    }
                    else
                    {
                        const int     lane = threadIdx.x & 31;
                        const double* ai =
                            q1.z >= 0 ? reinterpret_cast<const double*>(sm + q1.z) : a.ainv;
#pragma unroll 1
                        for(int row = warp; row < a.nc; row += kTailNT / 32)
                        {
                            double s = 0.0;
                            for(int k = lane; k < a.nc; k += 32)
                                s = fma(ai[(size_t)row * a.nc + k], (double)b[k], s);
                            s = warp_sum(s);
                            if(lane == 0)
                                x[row] = (T)s;
                        }
                    }
                }
                else if(q0.z == TAIL_SCALE)
                {
                    const T* b    = reinterpret_cast<const T*>(sm + q2.w);
                    const T* invd = reinterpret_cast<const T*>(sm + q3.x);
                    T*       z    = reinterpret_cast<T*>(sm + q3.y);
                    for(int i = threadIdx.x; i < q0.x; i += kTailNT)
                        z[i] = om * (invd[i] * b[i]);
                }
                else if(q0.w == TAIL_DCOL)
                    tail_rows<T, int16_t>(q0, q1, q2, q3, sm, om, dst);
                else if(q0.w == TAIL_COL)
                    tail_rows<T, int32_t>(q0, q1, q2, q3, sm, om, dst);
                else
                    tail_rows<T, void>(q0, q1, q2, q3, sm, om, dst);
            }
            __syncthreads();
        }
    }

    // Lays out one launch: shared-memory offsets, copies and passes.
    template <class T>
    struct tail_plan
    {
        tail_args a{};
        size_t    used = 0;

        int room(size_t bytes)
        {
            used += round16(bytes);
            return (int)(used - round16(bytes));
        }
        void copy(int off, const void* src, size_t bytes)
        {
            if(!bytes)
                return;
            a.copy[a.ncopy++] = tail_copy{src, off, (int)round16(bytes)};
            a.bytes += (int)round16(bytes);
        }
        // the operator of a pass; gathered: its columns are not needed
        tail_pass matrix(const lab_csr_impl* M, bool gathered)
        {
            tail_pass d{};
            const int ln = M->plan.lanes;
            d.m          = (int)M->m;
            // the W of launch_rowop's VECTOR dispatch (2, 4, 8, 16, else 32)
            d.lw   = M->plan.alg != LAB_SPMV_VECTOR ? 0
                     : ln == 2                      ? 1
                     : ln == 4                      ? 2
                     : ln == 8                      ? 3
                     : ln == 16                     ? 4
                                                    : 5;
            d.cols = gathered ? TAIL_GATHERED : M->lp.dcol ? TAIL_DCOL : TAIL_COL;
            d.y = d.z = -1;
            d.o_rp    = room((size_t)(M->m + 1) * 4);
            copy(d.o_rp, M->row_ptr, (size_t)(M->m + 1) * 4);
            const size_t nnz = (size_t)M->nnz;
            if(d.cols == TAIL_DCOL)
                copy(d.o_ci = room(nnz * 2), M->lp.dcol, nnz * 2);
            else if(d.cols == TAIL_COL)
                copy(d.o_ci = room(nnz * 4), M->col_ind, nnz * 4);
            d.o_v = room(nnz * sizeof(T));
            if constexpr(std::is_same<T, double>::value)
                copy(d.o_v, M->val, nnz * sizeof(T));
            else
                copy(d.o_v, M->lp.f32, nnz * sizeof(T));
            return d;
        }

        // edge: from level l's residual wr and iterate cur to its corrected iterate
        // dst; otherwise from level l + 1's right-hand side wr to its correction dst.
        void build(const hierarchy_impl* h, const lab_amg_options* o, int l, bool edge,
                   const T* wr, const T* cur, T* dst)
        {
            const int L = h->levels, nl = L - l;
            // level vectors x, t, b, r, D^-1
            int vec[kTailMax][5];
            for(int k = 0; k < nl; k++)
            {
                const lab_csr_impl* A  = h->A[l + 1 + k];
                const size_t        vb = (size_t)A->m * sizeof(T);
                for(int q = 0; q < 5; q++)
                    vec[k][q] = room(vb);
                if(k < nl - 1)
                    copy(vec[k][4], lv<T>::invd(A), vb);
            }
            a.nc     = (int)h->A[L]->m;
            a.a11    = (const double*)h->A[L]->val;
            a.ainv   = (const double*)h->coarse_inv;
            int ainv = -1;
            if(a.nc > 1 && a.nc <= 64)
                copy(ainv = room((size_t)a.nc * a.nc * sizeof(double)), a.ainv,
                     (size_t)a.nc * a.nc * sizeof(double));
            tail_pass A[kTailMax], R[kTailMax], P[kTailMax], Rp{}, Pp{};
            for(int k = 0; k < nl - 1; k++)
            {
                const int lk = l + 1 + k;
                A[k]         = matrix(h->A[lk], false);
                R[k]         = matrix(h->R[lk], false);
                P[k]         = matrix(h->P[lk], false);
            }
            int cx = 0;
            if(edge)
            {
                const lab_csr_impl* Rl = h->R[l];
                a.wr                   = wr;
                a.gci                  = Rl->col_ind;
                a.gnnz                 = (int)Rl->nnz;
                a.gx                   = room((size_t)Rl->nnz * sizeof(T));
                Rp                     = matrix(Rl, true);
                Pp                     = matrix(h->P[l], false);
                copy(cx = room((size_t)h->A[l]->m * sizeof(T)), cur,
                     (size_t)h->A[l]->m * sizeof(T));
            }
            else
                copy(vec[0][2], wr, (size_t)h->A[l + 1]->m * sizeof(T));

            // the passes; at[k]: which of x (0) and t (1) holds level k's iterate
            int  at[kTailMax] = {};
            auto add          = [&](const tail_pass& d, int mode) -> tail_pass& {
                a.pass[a.npass]      = d;
                a.pass[a.npass].mode = mode;
                return a.pass[a.npass++];
            };
            // b_k = R r; x_k = omega D^-1 b_k when k is not the coarsest (op_restrict with
            // the fused first sweep)
            auto restrict_to = [&](const tail_pass& R, int k, int in) {
                tail_pass& d = add(R, TAIL_RESTRICT);
                d.in         = in;
                d.y          = vec[k][2];
                if(k < nl - 1)
                {
                    d.z    = vec[k][0];
                    d.invd = vec[k][4];
                }
            };
            auto jacobi = [&](int k) {
                tail_pass& d = add(A[k], TAIL_JACOBI);
                d.in = d.x = vec[k][at[k]];
                d.b        = vec[k][2];
                d.invd     = vec[k][4];
                d.y        = vec[k][at[k] ^ 1];
                at[k] ^= 1;
            };
            if(edge)
                restrict_to(Rp, 0, a.gx);
            else if(nl > 1)
            {
                tail_pass& d = add(tail_pass{}, TAIL_SCALE);
                d.m          = (int)h->A[l + 1]->m;
                d.b          = vec[0][2];
                d.invd       = vec[0][4];
                d.z          = vec[0][0];
            }
            for(int k = 0; k < nl - 1; k++)
            {
                for(int it = 1; it < o->n1; it++)
                    jacobi(k);
                tail_pass& d = add(A[k], TAIL_RES);
                d.in         = vec[k][at[k]];
                d.b          = vec[k][2];
                d.y          = vec[k][3];
                restrict_to(R[k], k + 1, vec[k][3]);
            }
            {
                tail_pass& d = add(tail_pass{}, TAIL_COARSE);
                d.m          = a.nc;
                d.lw         = a.nc > 1 ? 5 : 0;
                d.b          = vec[nl - 1][2];
                d.y          = vec[nl - 1][0];
                d.o_v        = ainv;
            }
            for(int k = nl - 2; k >= 0; k--)
            {
                // x <- x + P e (op_prolong), into the other buffer
                tail_pass& d = add(P[k], TAIL_PROLONG);
                d.in         = vec[k + 1][at[k + 1]];
                d.x          = vec[k][at[k]];
                d.y          = vec[k][at[k] ^ 1];
                at[k] ^= 1;
                for(int it = 0; it < o->n2; it++)
                    jacobi(k);
            }
            if(edge)
            {
                tail_pass& d = add(Pp, TAIL_PROLONG);
                d.in         = vec[0][at[0]];
                d.x          = cx;
            }
            a.pass[a.npass - 1].out = 1;
            a.dst                   = dst;
            a.ndst                  = a.pass[a.npass - 1].m;
            a.omega                 = o->omega;
        }
    };

    // Levels l+1 .. L form a fused tail when the cycle is a V-cycle with Jacobi
    // smoothing (n1 >= 1) from a zero guess, level l's operators are not BF16, every
    // operator below l + 1 fits shared memory with the level vectors, and the
    // coarsest level is solved by a 1x1 division or a dense inverse of up to kTailInv
    // rows (every pass of the cycle in its own launch against the tail, us a cycle: 64
    // rows 10.7 / 9.1, 74 23.3 / 21.9, 82 11.9 / 11.3, 83 23.5 / 24.0, 98 11.6 / 13.1,
    // 170 12.6 / 17.0: one CTA reads all of the inverse).  One CTA stays
    // ahead of the 3 to 4 us that a separate launch costs up to about 16 entries per
    // thread and pass (kTailEntries).  R and P of level l join the launch up to
    // kTailEdge entries: above that one SM's share of the memory bandwidth costs more
    // than the two launches (9,433 entries: 25 us against 6).
    constexpr int64_t kTailEntries = 16 * kTailNT;
    constexpr int64_t kTailInv     = 80;

    int tail_ok(const hierarchy_impl* h, const lab_amg_options* o, int l)
    {
        const int L = h->levels, nl = L - l;
        if(o->cycle != LAB_CYCLE_V || o->smoother != LAB_SMOOTH_JACOBI || o->n1 < 1 ||
           l >= L || nl > kTailMax || level_bf16(o, l) || !h->status ||
           h->tail_off)
            return TAIL_NONE;
        const int64_t nc = h->A[L]->m;
        if(nc != 1 && !(nc > 1 && nc <= kTailInv && o->coarse == LAB_COARSE_DIRECT && h->coarse_inv))
            return TAIL_NONE;
        if(2 + (int64_t)(nl - 1) * (2 + (int64_t)o->n1 + std::max(o->n2, 0)) + 1 > kTailPasses)
            return TAIL_NONE;
        const size_t sz   = o->precision == LAB_PREC_FP64 ? 8 : 4;
        auto         fits = [](const lab_csr_impl* M, int64_t most) {
            return M && M->nnz <= most && M->m <= 8192 && M->plan.analysed;
        };
        auto bytes = [&](const lab_csr_impl* M) {
            return round16((size_t)(M->m + 1) * 4) + round16((size_t)M->nnz * 4) +
                   round16((size_t)M->nnz * sz);
        };
        size_t used = nc > 1 && nc <= 64 ? round16((size_t)nc * nc * 8) : 0;
        for(int k = l + 1; k <= L; k++)
        {
            if(!fits(h->A[k], kTailEntries))
                return TAIL_NONE;
            used += 5 * round16((size_t)h->A[k]->m * sz);
            if(k == L)
                break;
            if(!fits(h->R[k], kTailEntries) || !fits(h->P[k], kTailEntries))
                return TAIL_NONE;
            used += bytes(h->A[k]) + bytes(h->R[k]) + bytes(h->P[k]);
        }
        if(used > kTailSmem)
            return TAIL_NONE;
        if(!fits(h->R[l], kTailEdge) || !fits(h->P[l], kTailEdge))
            return nl > 1 ? TAIL_INNER : TAIL_NONE;
        used += 2 * bytes(h->R[l]) + bytes(h->P[l]) + round16((size_t)h->A[l]->m * sz);
        return used <= kTailSmem ? TAIL_EDGE : nl > 1 ? TAIL_INNER : TAIL_NONE;
    }

    template <class T>
    lab_status tail_launch(hierarchy_impl* h, int l, bool edge, const T* wr, const T* cur, T* dst,
                           const cyc_ctx& c)
    {
        tail_plan<T> t;
        t.build(h, c.o, l, edge, wr, cur, dst);
        t.a.skip     = c.skip;
        t.a.status   = h->status;
        t.a.timeouts = h->timeouts;
        t.a.polls    = h->wait_polls ? h->wait_polls : kStreamWaitLimit;
        t.a.held     = h->wait_held;
        static const cudaError_t attr = cudaFuncSetAttribute(
            k_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmem);
        LAB_CUDA(attr);
        LAB_LAUNCH(k_tail<T>, 1, kTailNT, t.used, c.s, t.a);
        return LAB_OK;
    }

    template lab_status tail_launch<double>(hierarchy_impl*, int, bool, const double*, const double*,
                                            double*, const cyc_ctx&);
    template lab_status tail_launch<float>(hierarchy_impl*, int, bool, const float*, const float*,
                                           float*, const cyc_ctx&);
}
