// Multigrid cycles (cycle.cu) as used by the solvers (solve.cu).
#pragma once

#include "amg.cuh"
#include "spmv_engine.cuh"

namespace lab
{
    struct cyc_ctx
    {
        const lab_amg_options* o;
        cudaStream_t           s;
        const int*             skip; // early-exit flag (PCG graph), may be null
    };

    // Allocate every per-level vector, analyse every operator, build the
    // reduced-precision copies / colourings / coarse inverse the options need.
    // Synchronises; never called inside a graph capture.
    lab_status cycle_prepare(hierarchy_impl* h, const lab_amg_options* o, cudaStream_t s);

    // Reads (and clears) the count of the cycles' waits that ran out: LAB_TIMEOUT if
    // there was one (its cycle's result is NaN).  Synchronises.
    lab_status cycle_check(hierarchy_impl* h, cudaStream_t s);

    // z = cycle(0; r) on level 0 (FP64 interface whatever the cycle precision).
    // With dot.out set, also (z, r) -> dot.out.  Enqueue only (capturable).
    lab_status cycle_precond(hierarchy_impl* h, const cyc_ctx& c, const double* r, double* z,
                             red_buf dot);
    // Reduced-precision preconditioner step of flexible PCG: the FP32 cycle on r,
    // (z, r) into zr.out and (z, q) into zq.out with z = fp64 of the cycle's result,
    // which stays in FP32 in the level-0 workspace (*z32; valid until the next cycle).
    lab_status cycle_precond_flex(hierarchy_impl* h, const cyc_ctx& c, const double* r,
                                  const double* q, red_buf zr, red_buf zq, const float** z32);

    // x <- cycle(x; b) on level 0 (stationary iteration step).  FP64 cycles run in
    // place; reduced-precision cycles run in correction form x += cycle(0; b - A x).
    lab_status cycle_iterate(hierarchy_impl* h, const cyc_ctx& c, const double* b, double* x);

    // Scalars and flags per system of a segmented PCG or column of a block one.
    enum
    {
        G_GAMMA = 0,
        G_PQ    = 1,
        G_RN    = 2,
        G_R0    = 3,
        G_GNEW  = 4,
        G_N     = 8
    };
    enum
    {
        GF_DONE   = 0,
        GF_ITER   = 1,
        GF_CONV   = 2,
        GF_STATUS = 3,
        GF_N      = 4
    };

    // Block vectors (cycle_blk.cu): ld columns interleaved per row.
    constexpr int     kBlkMax     = 64;  // columns solved together
    constexpr int64_t kBlkRedGrid = 592; // CTAs of a pass with a reduction (4 per SM)
    struct blk_red
    {
        double*       partial = nullptr; // kBlkRedGrid x ld
        unsigned int* counter = nullptr;
        double*       out     = nullptr; // column c's value at out[c * stride]
        int           stride  = 0;
        const int*    skip    = nullptr;
    };
    lab_status blk_from_columns(const double* x, int64_t ldx, int64_t n, int ncols, int ld,
                                double* xb, cudaStream_t s);
    lab_status blk_to_columns(const double* xb, int64_t n, int ncols, int ld, double* x,
                              int64_t ldx, cudaStream_t s);
    lab_status blk_norm(int64_t n, int ld, const double* r, const blk_red& red, cudaStream_t s);
    lab_status blk_init(double* sc, int* sf, int* gflags, int ld, int max_iter, cudaStream_t s);
    lab_status blk_update(int64_t n, int ld, double* x, double* r, const double* p, const double* q,
                          double* sc, int* sf, int* gflags, const blk_red& red, double rtol,
                          double atol, cudaStream_t s);
    lab_status blk_pupdate(int64_t n, int ld, double* p, const double* z, double* sc, int* sf,
                           int* gflags, unsigned int* counter, cudaStream_t s);
    lab_status blk_spmv_dot(const lab_csr_impl* A, int ld, const double* p, double* q,
                            const blk_red& red, cudaStream_t s);
    lab_status blk_residual(const lab_csr_impl* A, int ld, const double* x, const double* b,
                            double* r, cudaStream_t s);
    // Block V-cycle: whether the options are covered (V-cycle, Jacobi, FP64, 1x1 or
    // dense coarsest solve; call after cycle_prepare), the block workspace of at least ld
    // columns (outside graph capture; LAB_OOM also where it and vectors solve vectors of
    // level 0 are more than the hierarchy's bound), its release, unless it is small when
    // if_large is set, and z = cycle(0; r) on ld columns, with (z, r) per column into
    // dot.out when set.
    bool       cycle_block_supported(const hierarchy_impl* h, const lab_amg_options* o);
    lab_status cycle_prepare_block(hierarchy_impl* h, int ld, int vectors, cudaStream_t s);
    void       cycle_release_block(hierarchy_impl* h, bool if_large, cudaStream_t s);
    lab_status cycle_precond_block(hierarchy_impl* h, const cyc_ctx& c, int ld, const double* r,
                                   double* z, const blk_red& dot);

    // deterministic device reductions into r.out (grid <= kRedBlocks)
    lab_status dot_device(int64_t n, const double* x, const double* y, red_buf r, cudaStream_t s);
    lab_status norm_inf_device(int64_t n, const double* x, red_buf r, cudaStream_t s);
    unsigned   red_grid(int64_t n);
    unsigned   grid_for(int64_t n);

    // Per-precision views of a level's vectors and operator data.
    template <class T>
    struct lv;
    template <>
    struct lv<double>
    {
        static double* x(level_ws& w) { return w.x; }
        static double* b(level_ws& w) { return w.b; }
        static double* r(level_ws& w) { return w.r; }
        static double* t(level_ws& w) { return w.t; }
        static const double* invd(const lab_csr_impl* A) { return A->invdiag; }
    };
    template <>
    struct lv<float>
    {
        static float* x(level_ws& w) { return w.xf; }
        static float* b(level_ws& w) { return w.bf; }
        static float* r(level_ws& w) { return w.rf; }
        static float* t(level_ws& w) { return w.tf; }
        static const float* invd(const lab_csr_impl* A) { return A->lp.invd32; }
    };

    // BF16 value storage on the two finest levels (LAB_PREC_FP32_BF16).
    static inline bool level_bf16(const lab_amg_options* o, int l)
    {
        return o->precision == LAB_PREC_FP32_BF16 && l < 2;
    }

    // Fused tail (cycle_tail.cu): whether levels l+1 .. L of a V-cycle run as one launch,
    // with (EDGE) or without (INNER) the restriction out of level l and the prolongation
    // back, and that launch: from level l's residual wr and iterate cur to its corrected
    // iterate dst, or from level l+1's right-hand side wr to its correction dst.
    enum
    {
        TAIL_NONE,
        TAIL_INNER,
        TAIL_EDGE
    };
    int tail_ok(const hierarchy_impl* h, const lab_amg_options* o, int l);
    template <class T>
    lab_status tail_launch(hierarchy_impl* h, int l, bool edge, const T* wr, const T* cur, T* dst,
                           const cyc_ctx& c);

    __global__ void k_copy_d(double* __restrict__ y, const double* __restrict__ x, int64_t n,
                             const int* skip);
}
