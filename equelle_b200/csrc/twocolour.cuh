// Two-colour form of the multigrid-preconditioned BiCGStab (included by
// solver.cu, inside its anonymous namespace).
//
// On the cell graph of a Cartesian grid every level of the hierarchy takes
// two colours: the red block rows [0, nr) and the black ones [nr, nb), with
// no couplings inside a colour.  Red unknowns can then be eliminated exactly,
//   x_r = D_r^-1 (b_r - U x_b),   S x_b = b_b - L b_r,   S = A_bb - L U,
// with L = A_br D_r^-1 and U = A_rb the off-diagonal blocks of the block
// ILU(0) factors and A_bb the black diagonal blocks, so that BiCGStab runs on
// the black half: vectors of half the length, and S x as two half products
// (y = -U x, A_bb x + L y) that read each stored block of the factors once.
// The residual of the whole system is that of its black half (red rows are
// solved exactly), so the convergence test is unchanged.
//
// The V-cycle's block ILU(0) sweeps read the same factors (D_b is the black
// diagonal block of the factorization, A_bb - the diagonal blocks of L U).
// With right-hand side (r_r, r_b) and iterate z_b,
//   y   = r_r - U z_b                       (rb_y_rows)
//   t_b = r_b - A_bb z_b - L y              (the residual; red rows: 0)
//   z_b += D_b^-1 t_b                       (rb_post_rows)
//   z_r = D_r^-1 (r_r - U z_b)              (rb_fin_rows)
// is one sweep from any z_b: the red part of the iterate is never needed
// before the last line, the residual of the down-leg is summed straight into
// the coarse right-hand side (rb_res_rows), and the coarse level's last two
// steps add alpha times their rows to the fine black rows (scatter_up).  A
// level with pre-smoothing takes six half products of its factors, one
// without (Level::pre) three; the level-0 cycle needs no red rows at all.
//
// Bound: HBM on the fine levels (the factors, 36 bytes per 2 x 2 FP64 block),
// latency of dependent steps on the coarse ones.  Measured on one time step
// against the full-length form over stages (two sweeps, residual, A P up-leg
// and a full product per application; 2 x 2 x 2 aggregates only): two-phase
// 128x128x64, 203 BiCGStab iterations of 0.74 ms -> 90 of 0.65 ms (the
// iterations by aggregation along z alone on the first two levels); 512x512,
// 53 of 0.50 ms -> 52 of 0.32 ms; 33x31x17, 117 of 0.175 -> 58 of 0.167 ms.

// Where a level's finished rows go: alpha z is added to (add) or stored in
// the black members, g per block row of this level, of the finer level's z.
struct UpView {
    const int* list = nullptr;
    int g = 0;
    int add = 0;
    double alpha = 1.0;
    double* w = nullptr;  // finer level's z, indexed by its block rows; null: no finer level
};

template <int B, bool CG>
__device__ __forceinline__ void scatter_up(const UpView& u, int R, const double (&z)[B])
{
    if (u.w == nullptr) return;
    for (int s = 0; s < u.g; ++s) {
        const int m = u.list[R * u.g + s];
        if (m < 0) continue;
        double f[B];
#pragma unroll
        for (int c = 0; c < B; ++c) f[c] = 0.0;
        if (u.add) load_bvec<B, double, CG>(u.w, m, f);
#pragma unroll
        for (int c = 0; c < B; ++c) f[c] += u.alpha * z[c];
        store_bvec<B, double>(u.w, m, f);
    }
}

// The steps below are loops over a row range for thread `tid` of `nth`,
// shared by the one-step kernels and the fused coarse cycle (see
// mg_tail_kernel), so that both compute every element alike.  Vectors are
// indexed by block row; r == null stands for a zero red right-hand side.

// y_R = r_R - sum U_RJ z_J over the red rows.
template <int B, int KM, class M, bool CG, bool U>
__device__ __forceinline__ void rb_y_rows(int nr, const SellView& m, const M* __restrict__ lu, const double* r,
                                          const double* z, double* y, int tid, int nth)
{
    for (int R = tid; R < nr; R += nth) {
        double acc[B];
#pragma unroll
        for (int c = 0; c < B; ++c) acc[c] = 0.0;
        bdot<B, KM, double, M, CG, U>(m, slice_base<U>(m, R), R & 31, 1, m.len[R], lu, z, z, INT_MAX, acc);
        double v[B];
#pragma unroll
        for (int c = 0; c < B; ++c) v[c] = 0.0;
        if (r) load_bvec<B, double, CG>(r, R, v);
#pragma unroll
        for (int c = 0; c < B; ++c) v[c] -= acc[c];
        store_bvec<B, double>(y, R, v);
    }
}

// z_R = D_R^-1 (r_R - sum U_RJ z_J) over the red rows, handed to the finer
// level (a level's red rows are read by nothing else).
template <int B, int KM, class M, bool CG, bool U>
__device__ __forceinline__ void rb_fin_rows(int nr, const SellView& m, const M* __restrict__ lu, const double* r,
                                            const double* z, const UpView& up, int tid, int nth)
{
    for (int R = tid; R < nr; R += nth) {
        const int lane = R & 31, sb = slice_base<U>(m, R);
        double acc[B];
#pragma unroll
        for (int c = 0; c < B; ++c) acc[c] = 0.0;
        bdot<B, KM, double, M, CG, U>(m, sb, lane, 1, m.len[R], lu, z, z, INT_MAX, acc);
        double v[B], x[B];
        load_bvec<B, double, CG>(r, R, v);
#pragma unroll
        for (int c = 0; c < B; ++c) v[c] -= acc[c];
        bmatvec<B, M>(lu, sb, lane, v, x);
        scatter_up<B, CG>(up, R, x);
    }
}

// z_R = D_R^-1 (r_R - sum L_RJ y_J) over the black rows, y the red
// right-hand side (null: zero): the sweep from z = 0.
template <int B, int KM, class M, bool CG, bool U>
__device__ __forceinline__ void rb_pre_rows(int nr, int nb, const SellView& m, const M* __restrict__ lu,
                                            const double* r, const double* y, double* z, int tid, int nth)
{
    for (int R = (nr & ~31) + tid; R < nb; R += nth) {  // whole slices
        if (R < nr) continue;
        const int lane = R & 31, sb = slice_base<U>(m, R), d = m.len[R] - 1;
        double acc[B];
#pragma unroll
        for (int c = 0; c < B; ++c) acc[c] = 0.0;
        if (y) bdot<B, KM, double, M, CG, U>(m, sb, lane, 0, d, lu, y, y, INT_MAX, acc);
        double v[B], x[B];
        load_bvec<B, double, CG>(r, R, v);
#pragma unroll
        for (int c = 0; c < B; ++c) v[c] -= acc[c];
        bmatvec<B, M>(lu, sb + (d << 5), lane, v, x);
        store_bvec<B, double>(z, R, x);
    }
}

// t_R = r_R - A_RR z_R - sum L_RJ y_J of one black row.
template <int B, int KM, class M, bool CG, bool U>
__device__ __forceinline__ void rb_residual_row(int R, const SellView& m, const M* __restrict__ a,
                                                const M* __restrict__ lu, const double* r, const double* y,
                                                const double (&z)[B], double (&t)[B])
{
    const int lane = R & 31, sb = slice_base<U>(m, R), d = m.len[R] - 1;
    double acc[B], az[B];
#pragma unroll
    for (int c = 0; c < B; ++c) acc[c] = 0.0;
    bdot<B, KM, double, M, CG, U>(m, sb, lane, 0, d, lu, y, y, INT_MAX, acc);
    bmatvec<B, M>(a, sb + (d << 5), lane, z, az);
    load_bvec<B, double, CG>(r, R, t);
#pragma unroll
    for (int c = 0; c < B; ++c) t[c] = (t[c] - az[c]) - acc[c];
}

// rc_P = sum of t over the black members of aggregate P, g lanes per
// aggregate (a power of two; member s of P at list[P g + s], -1 past the
// last): the lanes' rows are consecutive between neighbouring aggregates, so
// a warp reads whole segments, and the sum is a butterfly over the g lanes.
template <int B, int KM, class M, bool CG, bool U>
__device__ __forceinline__ void rb_res_rows(int ncb, int g, const int* __restrict__ list, const SellView& m,
                                            const M* __restrict__ a, const M* __restrict__ lu, const double* r,
                                            const double* y, const double* z, double* rc, int tid, int nth)
{
    const int items = ncb * g, padded = (items + 31) & ~31;
    for (int i = tid; i < padded; i += nth) {
        const int R = i < items ? list[i] : -1;
        double t[B];
#pragma unroll
        for (int c = 0; c < B; ++c) t[c] = 0.0;
        if (R >= 0) {
            double zv[B];
            load_bvec<B, double, CG>(z, R, zv);
            rb_residual_row<B, KM, M, CG, U>(R, m, a, lu, r, y, zv, t);
        }
        for (int o = 1; o < g; o <<= 1)
#pragma unroll
            for (int c = 0; c < B; ++c) t[c] += __shfl_xor_sync(0xffffffffu, t[c], o);
        if (i < items && (i & (g - 1)) == 0) store_bvec<B, double>(rc, i / g, t);
    }
}

// rc_P = sum of r over the members of aggregate P in `list`, g per aggregate.
template <int B, bool CG>
__device__ __forceinline__ void rb_restrict_rows(int ncb, int g, const int* __restrict__ list, const double* r,
                                                 double* rc, int tid, int nth)
{
    for (int P = tid; P < ncb; P += nth) {
        double s[B];
#pragma unroll
        for (int c = 0; c < B; ++c) s[c] = 0.0;
        for (int k = 0; k < g; ++k) {
            const int m = list[P * g + k];
            if (m < 0) continue;
            double v[B];
            load_bvec<B, double, CG>(r, m, v);
#pragma unroll
            for (int c = 0; c < B; ++c) s[c] += v[c];
        }
        store_bvec<B, double>(rc, P, s);
    }
}

// z_R += D_R^-1 (r_R - A_RR z_R - sum L_RJ y_J) over the black rows, handed
// to the finer level.
template <int B, int KM, class M, bool CG, bool U>
__device__ __forceinline__ void rb_post_rows(int nr, int nb, const SellView& m, const M* __restrict__ a,
                                             const M* __restrict__ lu, const double* r, const double* y, double* z,
                                             const UpView& up, int tid, int nth)
{
    for (int R = (nr & ~31) + tid; R < nb; R += nth) {  // whole slices
        if (R < nr) continue;
        double zv[B], t[B], x[B];
        load_bvec<B, double, CG>(z, R, zv);
        rb_residual_row<B, KM, M, CG, U>(R, m, a, lu, r, y, zv, t);
        bmatvec<B, M>(lu, slice_base<U>(m, R) + ((m.len[R] - 1) << 5), R & 31, t, x);
#pragma unroll
        for (int c = 0; c < B; ++c) zv[c] += x[c];
        store_bvec<B, double>(z, R, zv);
        scatter_up<B, CG>(up, R, zv);
    }
}

// The coarsest level: z = inv r, a warp per unknown (see dense_rows), handed
// to the finer level.
template <int B, class M, bool CG>
__device__ __forceinline__ void rb_dense_rows(int n, const M* __restrict__ inv, const double* r, const UpView& up,
                                              int tid, int nth)
{
    const int lane = tid & 31;
    for (int i = tid >> 5; i < n; i += nth >> 5) {
        double s = 0.0;
        for (int j = lane; j < n; j += 32) s += (double)inv[i * n + j] * (CG ? __ldcg(r + j) : r[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const int P = i / B, c = i - P * B;
        if (lane < up.g) {
            const int m = up.list[P * up.g + lane];
            if (m >= 0) {
                double* w = up.w + (size_t)m * B + c;
                const double f = up.add ? (CG ? __ldcg(w) : *w) : 0.0;
                *w = f + up.alpha * s;
            }
        }
    }
}

// ---- one step per launch ------------------------------------------------------
template <int B, int KM, class M>
__global__ void __launch_bounds__(512) rb_y_kernel(int nr, SellView m, const M* __restrict__ lu, const double* r,
                                                   const double* z, double* y, const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_y_rows<B, KM, M, false, false>(nr, m, lu, r, z, y, tid, nth);
}

template <int B, int KM, class M>
__global__ void __launch_bounds__(512) rb_fin_kernel(int nr, SellView m, const M* __restrict__ lu, const double* r,
                                                     const double* z, UpView up, const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_fin_rows<B, KM, M, false, false>(nr, m, lu, r, z, up, tid, nth);
}

template <int B, int KM, class M>
__global__ void __launch_bounds__(512) rb_pre_kernel(int nr, int nb, SellView m, const M* __restrict__ lu,
                                                     const double* r, const double* y, double* z, const KScal* sc,
                                                     int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_pre_rows<B, KM, M, false, false>(nr, nb, m, lu, r, y, z, tid, nth);
}

template <int B, int KM, class M>
__global__ void __launch_bounds__(512) rb_res_kernel(int ncb, int g, const int* __restrict__ list, SellView m,
                                                     const M* __restrict__ a, const M* __restrict__ lu,
                                                     const double* r, const double* y, const double* z, double* rc,
                                                     const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_res_rows<B, KM, M, false, false>(ncb, g, list, m, a, lu, r, y, z, rc, tid, nth);
}

template <int B>
__global__ void rb_restrict_kernel(int ncb, int g, const int* __restrict__ list, const double* r, double* rc,
                                   const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_restrict_rows<B, false>(ncb, g, list, r, rc, tid, nth);
}

template <int B, int KM, class M>
__global__ void __launch_bounds__(512) rb_post_kernel(int nr, int nb, SellView m, const M* __restrict__ a,
                                                      const M* __restrict__ lu, const double* r, const double* y,
                                                      double* z, UpView up, const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_post_rows<B, KM, M, false, false>(nr, nb, m, a, lu, r, y, z, up, tid, nth);
}

template <int B, class M>
__global__ void rb_dense_kernel(int n, const M* __restrict__ inv, const double* r, UpView up, const KScal* sc,
                                int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    rb_dense_rows<B, M, false>(n, inv, r, up, (int)threadIdx.x, (int)blockDim.x);
}

// ---- BiCGStab on the black half ------------------------------------------------
// g = b_b - L b_r is the first residual; with the vectors' start values, the
// shadow residual, and the dots of bicg_init (rr of g, thr of the whole b).
// b is in block-row order; the other vectors hold the black rows only.
template <int B, int KM>
__global__ void __launch_bounds__(kThreads) rb_init_kernel(int nr, int nb, SellView m, const double* __restrict__ lu,
                                                           const double* __restrict__ b, double* r, double* rhat,
                                                           double* p, double* v, double* x, double* partials,
                                                           unsigned int* counter, KScal* sc, double tol2)
{
    double d[3] = {0.0, 0.0, 0.0};
    GRID_STRIDE(rr, nb)
    {
        const int R = (int)rr;
        double bv[B];
        load_bvec<B, double>(b, R, bv);
#pragma unroll
        for (int c = 0; c < B; ++c) d[2] += bv[c] * bv[c];
        if (R < nr) continue;
        double acc[B];
#pragma unroll
        for (int c = 0; c < B; ++c) acc[c] = 0.0;
        bdot<B, KM, double, double>(m, m.slice_ptr[R >> 5], R & 31, 0, m.len[R] - 1, lu, b, b, INT_MAX, acc);
        const int q = R - nr;
#pragma unroll
        for (int c = 0; c < B; ++c) {
            const int64_t i = (int64_t)q * B + c;
            const double gi = bv[c] - acc[c], hi = shadow_entry(i);
            r[i] = gi;
            rhat[i] = hi;
            p[i] = 0.0;
            v[i] = 0.0;
            x[i] = 0.0;
            d[0] += gi * gi;
            d[1] += hi * gi;
        }
    }
    double s[3];
    if (grid_sum<3>(d, partials, counter, s)) {
        sc->rho = 1.0;
        sc->alpha = 1.0;
        sc->omega = 1.0;
        sc->rho_new = s[1];
        sc->rr = s[0];
        sc->thr = tol2 * s[2];
        sc->s_conv = 0;
        sc->iterations = 0;
        sc->status = s[0] <= sc->thr ? ST_CONV : ST_RUN;
    }
}

// v = S z = A_bb z + L y (y = -U z) over the black rows, with the dots of
// bicg_spmv_alpha (OMEGA false: alpha = rho_new / (h . v), h the shadow
// residual) or bicg_spmv_omega (omega = (v . h) / (v . v), h = s).  z, h and
// v hold the black rows only.
template <int B, int KM, bool OMEGA>
__global__ void __launch_bounds__(kThreads)
    rb_spmv_kernel(int nr, int nb, SellView m, const double* __restrict__ a, const double* __restrict__ lu,
                   const double* __restrict__ z, const double* __restrict__ y, const double* __restrict__ h,
                   double* __restrict__ v, double* partials, unsigned int* counter, KScal* sc)
{
    pdl_wait();
    if (stopped(sc) || (OMEGA && sc->s_conv)) return;
    constexpr int ND = OMEGA ? 2 : 1;
    double d[ND];
#pragma unroll
    for (int k = 0; k < ND; ++k) d[k] = 0.0;
    GRID_STRIDE(i, nb - (nr & ~31))  // whole slices
    {
        const int R = (nr & ~31) + (int)i, q = R - nr;
        if (q < 0) continue;
        const int lane = R & 31, sb = m.slice_ptr[R >> 5], dk = m.len[R] - 1;
        double acc[B], zv[B], az[B], hv[B];
#pragma unroll
        for (int c = 0; c < B; ++c) acc[c] = 0.0;
        bdot<B, KM, double, double>(m, sb, lane, 0, dk, lu, y, y, INT_MAX, acc);
        load_bvec<B, double>(z, q, zv);
        bmatvec<B, double>(a, sb + (dk << 5), lane, zv, az);
        load_bvec<B, double>(h, q, hv);
#pragma unroll
        for (int c = 0; c < B; ++c) acc[c] += az[c];
        store_bvec<B, double>(v, q, acc);
#pragma unroll
        for (int c = 0; c < B; ++c) {
            d[0] += hv[c] * acc[c];
            if (OMEGA) d[ND - 1] += acc[c] * acc[c];
        }
    }
    double s[ND];
    if (grid_sum<ND>(d, partials, counter, s)) {
        if (OMEGA) {
            sc->ts = s[0];
            sc->tt = s[ND - 1];
            if (s[ND - 1] == 0.0 || !isfinite(s[ND - 1])) sc->status = ST_BREAK;
            else sc->omega = s[0] / s[ND - 1];
        } else {
            sc->rv = s[0];
            if (s[0] == 0.0 || !isfinite(s[0])) sc->status = ST_BREAK;
            else sc->alpha = sc->rho_new / s[0];
        }
    }
}

// The solution in the natural unknown order: x_b, and x_r = D_r^-1 (b_r - U x_b).
template <int B, int KM>
__global__ void __launch_bounds__(kThreads) rb_solution_kernel(int nr, int nb, SellView m,
                                                               const double* __restrict__ lu,
                                                               const double* __restrict__ b,
                                                               const double* __restrict__ x,
                                                               const int* __restrict__ perm, double* __restrict__ out)
{
    GRID_STRIDE(rr, nb)
    {
        const int R = (int)rr;
        double z[B];
        if (R < nr) {
            const int lane = R & 31, sb = m.slice_ptr[R >> 5];
            double acc[B], v[B];
#pragma unroll
            for (int c = 0; c < B; ++c) acc[c] = 0.0;
            const double* xs = x - (int64_t)nr * B;
            bdot<B, KM, double, double>(m, sb, lane, 1, m.len[R], lu, xs, xs, INT_MAX, acc);
            load_bvec<B, double>(b, R, v);
#pragma unroll
            for (int c = 0; c < B; ++c) v[c] -= acc[c];
            bmatvec<B, double>(lu, sb, lane, v, z);
        } else {
            load_bvec<B, double>(x, R - nr, z);
        }
#pragma unroll
        for (int c = 0; c < B; ++c) out[perm[R * B + c]] = z[c];
    }
}

// ---- the coarse end of the cycle in one kernel ----------------------------------
// As mg_tail_kernel: one thread-block cluster, a cluster barrier between the
// steps, the coarsest levels in block 0's shared memory.
struct RbLocal {
    int a, lu, inv, col, len, list, r, w;
};

template <class M>
struct RbTailLevel {
    int nb = 0, nr = 0, n = 0, coarsest = 0, pre = 1;
    int g = 0;                   // members per aggregate in `list`
    SellView m{};
    const M* a = nullptr;
    const M* lu = nullptr;
    const M* inv = nullptr;      // coarsest level
    const int* list = nullptr;   // members restricted to the next level (black ones when pre)
    const double* r = nullptr;   // right-hand side by block row
    const double* r_red = nullptr;  // the same, or null where its red rows are zero
    double* rw = nullptr;        // where the finer level's restriction writes r
    double* z = nullptr;         // black rows of the iterate, by block row
    double* y = nullptr;         // red rows' work vector, by block row
    UpView up;                   // where its rows go
    RbLocal so{};
};

template <class M>
struct RbTailParams {
    RbTailLevel<M> lv[kMaxTail];
    int nlev = 0;
    int local_first = kMaxTail;
    int nregions = 0;
    int ncopies = 0;
    PrefetchRegion reg[kMaxPrefetch];
    TailCopy copies[kMaxCopies];
    long long* trace = nullptr;
};
static_assert(sizeof(RbTailParams<double>) <= 4096, "fused cycle parameters exceed 4 KB");

// One level's steps down to its coarse right-hand side; `sync` ends a step.
template <int B, int KM, class M, bool CG, class Sync>
__device__ __forceinline__ void rb_down(const RbTailLevel<M>& L, const SellView& m, const M* a, const M* lu,
                                        const int* list, const double* r, const double* r_red, double* z, double* y,
                                        int ncb, double* rc, int tid, int nth, Sync&& sync)
{
    constexpr bool U = KM > 0;
    if (L.pre) {
        rb_pre_rows<B, KM, M, CG, U>(L.nr, L.nb, m, lu, r, r_red, z, tid, nth);
        sync();
        rb_y_rows<B, KM, M, CG, U>(L.nr, m, lu, r_red, z, y, tid, nth);
        sync();
        rb_res_rows<B, KM, M, CG, U>(ncb, L.g, list, m, a, lu, r, y, z, rc, tid, nth);
    } else {
        rb_restrict_rows<B, CG>(ncb, L.g, list, r, rc, tid, nth);
    }
    sync();
}

template <int B, int KM, class M, bool CG, class Sync>
__device__ __forceinline__ void rb_up(const RbTailLevel<M>& L, const SellView& m, const M* a, const M* lu,
                                      const double* r, const double* r_red, double* z, double* y, const UpView& up,
                                      int tid, int nth, Sync&& sync)
{
    constexpr bool U = KM > 0;
    rb_y_rows<B, KM, M, CG, U>(L.nr, m, lu, r_red, z, y, tid, nth);
    sync();
    rb_post_rows<B, KM, M, CG, U>(L.nr, L.nb, m, a, lu, r, y, z, up, tid, nth);
    if (up.w == nullptr) return;
    sync();
    rb_fin_rows<B, KM, M, CG, U>(L.nr, m, lu, r, z, up, tid, nth);
    sync();
}

// The levels from lf on, on block 0 alone, in its shared memory; the
// correction goes to level lf - 1's z in global memory.
template <int B, int KM, class M>
__device__ void rb_local_cycle(const RbTailParams<M>& p, int lf, unsigned char* sm)
{
    const int tid = (int)threadIdx.x, nth = (int)blockDim.x;
    auto sync = [] { __syncthreads(); };
    auto at_r = [&](int l) { return (double*)(sm + p.lv[l].so.r); };
    auto at_w = [&](int l) { return (double*)(sm + p.lv[l].so.w); };
    auto view = [&](int l) {
        const RbLocal& o = p.lv[l].so;
        return SellView{nullptr, (const int*)(sm + o.col), (const int*)(sm + o.len), nullptr, p.lv[l].m.width};
    };
    // where level l's rows go: the level above it in shared memory, or
    // level lf - 1 in global memory
    auto up_of = [&](int l) {
        UpView u = p.lv[l].up;
        if (l > lf) {
            u.list = (const int*)(sm + p.lv[l - 1].so.list);
            if (!p.lv[l - 1].pre) u.list = p.lv[l].up.list;
            u.w = at_w(l - 1);
        }
        return u;
    };
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (int i = tid; i < p.lv[lf].n; i += nth) at_r(lf)[i] = __ldcg(p.lv[lf].r + i);
    __syncthreads();
    int l = lf;
    for (; !p.lv[l].coarsest; ++l) {
        const RbTailLevel<M>& L = p.lv[l];
        rb_down<B, KM, M, false>(L, view(l), (const M*)(sm + L.so.a), (const M*)(sm + L.so.lu),
                                 (const int*)(sm + L.so.list), at_r(l), at_r(l), at_w(l), at_w(l), p.lv[l + 1].nb,
                                 at_r(l + 1), tid, nth, sync);
    }
    rb_dense_rows<B, M, false>(p.lv[l].n, (const M*)(sm + p.lv[l].so.inv), at_r(l), up_of(l), tid, nth);
    __syncthreads();
    for (--l; l >= lf; --l) {
        const RbTailLevel<M>& L = p.lv[l];
        rb_up<B, KM, M, false>(L, view(l), (const M*)(sm + L.so.a), (const M*)(sm + L.so.lu), at_r(l), at_r(l),
                               at_w(l), at_w(l), up_of(l), tid, nth, sync);
    }
}

template <int B, int KM, class M>
__global__ void __launch_bounds__(kTailThreads)
    rb_tail_kernel(const __grid_constant__ RbTailParams<M> p, const KScal* sc, int skip_if_s)
{
    extern __shared__ __align__(16) unsigned char tail_smem[];
    // constant during a solve: fetched before the wait for the previous kernel
    const int lf = p.local_first < p.nlev ? p.local_first : p.nlev;
    if (lf < p.nlev && blockIdx.x == 0) start_local_copies(p.copies, p.ncopies, tail_smem);
    prefetch_regions(p.reg, p.nregions);
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    long long* const trace = p.trace;
    int tk = 0;
    if (trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0) trace[tk] = clock64();
    ++tk;
    auto sync = [&] { tail_step(trace, tk); };
    // a warp (one slice of 32 rows) at a time, round robin over the blocks
    const int tid = (((int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x) << 5) | (int)(threadIdx.x & 31);
    const int nth = (int)(gridDim.x * blockDim.x);
    int l = 0;
    for (; l < lf && !p.lv[l].coarsest; ++l) {
        const RbTailLevel<M>& L = p.lv[l];
        rb_down<B, KM, M, true>(L, L.m, L.a, L.lu, L.list, L.r, L.r_red, L.z, L.y, p.lv[l + 1].nb, p.lv[l + 1].rw,
                                tid, nth, sync);
    }
    if (l == lf) {
        // block 0 alone; the other blocks wait at the next cluster barrier
        if constexpr (KM > 0) {
            if (blockIdx.x == 0) rb_local_cycle<B, KM, M>(p, lf, tail_smem);
        }
    } else {
        rb_dense_rows<B, M, true>(p.lv[l].n, p.lv[l].inv, p.lv[l].r, p.lv[l].up, tid, nth);
    }
    sync();
    for (--l; l >= 0; --l) {
        const RbTailLevel<M>& L = p.lv[l];
        rb_up<B, KM, M, true>(L, L.m, L.a, L.lu, L.r, L.r_red, L.z, L.y, L.up, tid, nth, sync);
    }
}
