// Two-colour form of the multigrid-preconditioned BiCGStab on the seven-point
// (five-point) block stencils of Cartesian grids (included by solver.cu,
// inside its anonymous namespace).
//
// Colouring the cells by the parity of i + j + k, no two cells of a colour
// are coupled, so the red unknowns can be eliminated exactly,
//   x_r = D_r^-1 (b_r - U x_b),   S x_b = b_b - L b_r,   S = A_bb - L U,
// with L = A_br D_r^-1 and U = A_rb the off-diagonal blocks of the block
// ILU(0) factors, D_r = A_rr, and A_bb the black diagonal blocks, so that
// BiCGStab runs on the black half: vectors of half the length, and S x as two
// half products (y = -U x, A_bb x + L y) that read each stored block once.
// The residual of the whole system is that of its black half (red rows are
// solved exactly), so the convergence test is unchanged.
//
// The V-cycle's block ILU(0) sweeps read the same factors (D_b, the black
// diagonal block of the factorization, is A_bb less the diagonal blocks of
// L U).  With right-hand side (r_r, r_b) and iterate z_b,
//   y   = r_r - U z_b                       (rb_y_rows)
//   t_b = r_b - A_bb z_b - L y              (the residual; red rows: 0)
//   z_b += D_b^-1 t_b                       (rb_post_rows)
//   z_r = D_r^-1 (r_r - U z_b)              (rb_fin_rows)
// is one sweep from any z_b: the red part of the iterate is never needed
// before the last line, the residual of the down-leg is summed straight into
// the coarse right-hand side (rb_res_rows), and the coarse level's last two
// steps add alpha times their rows to the fine black cells (scatter_up).  A
// level with pre-smoothing (Level::pre) takes six half products of its
// factors, one without three; level 0 needs no red rows at all.
//
// Layout: cell c = i + nx (j + ny k) is number c >> 1 of its colour whatever
// the sides (lines, planes or the whole grid alternate), so a neighbour's
// place follows from index arithmetic: no column indices, row lengths or
// slices are stored or waited for, and a step's loads (blocks and gathered
// vector) are one round trip.  Blocks are stored by direction (W, E, S, N, B,
// T), each direction contiguous over the rows of a colour: a warp's loads are
// whole segments.  Couplings that the Jacobian's pattern lacks are zero
// blocks.
//
// Bound: HBM on the fine levels (32 bytes per 2 x 2 FP64 block), latency of
// dependent steps on the coarse ones.  Measured on one time step, against the
// full-length form over stages with 2 x 2 x 2 aggregates only and against
// this form on the block sliced layout (stored columns and lengths): Krylov
// time of two-phase 128x128x64, 150 (203 iterations) -> 59 -> 51 ms (90; the
// iterations by pairing along z alone on the first two levels); 512x512, 26.5
// -> 16.6 -> 11.6 ms; 33x31x17, 20.6 -> 9.7 -> 7.9 ms; impes 97x83x41, 31.6 ->
// 12.6 -> 10.4 ms.  First step of a new 128x128x64 runtime, with the analysis
// on the host, then on the device: 526 -> 180 ms.

// Division by a run-time constant, exact for 0 <= n < 2^31: with l =
// ceil(log2 d) and m = floor(2^(31+l) / d) + 1, floor(n / d) = floor(n m /
// 2^(31+l)) since m d - 2^(31+l) <= d <= 2^l (Granlund and Montgomery 1994).
struct FastDiv {
    unsigned m = 0;
    int s = 0;  // < 0: d is 1
    FastDiv() = default;
    explicit FastDiv(unsigned d)
    {
        int l = 0;
        while ((1ull << l) < d) ++l;
        m = (unsigned)((1ull << (31 + l)) / d + 1);
        s = l - 1;
    }
    __device__ __forceinline__ int operator()(int n) const { return s < 0 ? n : (int)(__umulhi((unsigned)n, m) >> s); }
};

// A level's grid of cells.
struct RbGrid {
    int nx = 1, ny = 1, nz = 1, n = 1, nr = 1;  // cells, red cells
    int step = 1;                               // cells of a plane
    FastDiv by_x, by_plane;
    RbGrid() = default;
    RbGrid(int x, int y, int z) : nx(x), ny(y), nz(z), n(x * y * z), nr((n + 1) / 2), step(x * y), by_x(x), by_plane(x * y) {}
};

struct Cell {
    int c, i, j, k;
};

__device__ __forceinline__ Cell cell_at(const RbGrid& g, int c)
{
    Cell e;
    e.c = c;
    e.k = g.by_plane(c);
    const int r = c - e.k * g.step;
    e.j = g.by_x(r);
    e.i = r - e.j * g.nx;
    return e;
}

// Cell number q of a colour (0 red, 1 black): the one of 2 q and 2 q + 1 of
// that colour.
__device__ __forceinline__ Cell cell_of(const RbGrid& g, int colour, int q)
{
    Cell e = cell_at(g, 2 * q);
    if (((e.i + e.j + e.k) & 1) != colour) {
        ++e.c;
        if (++e.i == g.nx) {
            e.i = 0;
            if (++e.j == g.ny) {
                e.j = 0;
                ++e.k;
            }
        }
    }
    return e;
}

// Whether the cell has a neighbour in direction d, and that neighbour's
// number in the other colour.
__device__ __forceinline__ bool neighbour(const RbGrid& g, const Cell& e, int d, int& q)
{
    const int off = d < 2 ? 1 : d < 4 ? g.nx : g.step;
    q = (d & 1 ? e.c + off : e.c - off) >> 1;
    switch (d) {
    case 0: return e.i > 0;
    case 1: return e.i + 1 < g.nx;
    case 2: return e.j > 0;
    case 3: return e.j + 1 < g.ny;
    case 4: return e.k > 0;
    default: return e.k + 1 < g.nz;
    }
}

// The arrays of a level's matrix, one after the other: off-diagonal blocks of
// the red and of the black cells by direction, diagonal blocks of the red
// cells and of the black ones, and the factors' black diagonal blocks.  As
// gathered from the Jacobian: A.  As factored: U (unchanged), L, D_r^-1,
// A_bb (unchanged), D_b^-1.
template <class M>
struct RbMatrix {
    M *U, *L, *dr, *abb, *db;
    __host__ __device__ RbMatrix(M* base, int nd, int bb, int n, int nr)
    {
        U = base;
        L = U + (size_t)nd * nr * bb;
        dr = L + (size_t)nd * (n - nr) * bb;
        abb = dr + (size_t)nr * bb;
        db = abb + (size_t)(n - nr) * bb;
    }
    static size_t values(int nd, int bb, int n, int nr) { return ((size_t)(nd + 1) * n + (n - nr)) * bb; }
};

// acc += sum over the neighbours of A_d x_d, directions in order, row q of
// `rows`.  The loads are unconditional, so that all of them are issued before
// the first sum (with a branch per neighbour the compiler waited for each one
// in turn, in 34 registers): the block of a missing neighbour is stored as
// zero, and the vector is then read at the row's own number, or the last one.
template <int B, int ND, class M, bool CG>
__device__ __forceinline__ void stencil_dot(const RbGrid& g, const Cell& e, int q, int rows, const M* __restrict__ a,
                                            const double* __restrict__ x, double (&acc)[B])
{
    constexpr int BB = B * B;
    M av[ND][BB];
    double xv[ND][B];
    const int own = min(q, g.n - rows - 1);  // the other colour has n - rows cells
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        int nq;
        if (!neighbour(g, e, d, nq)) nq = own;
        load_block<BB, M>(a + ((size_t)d * rows + q) * BB, av[d]);
        load_bvec<B, double, CG>(x, nq, xv[d]);
    }
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int i = 0; i < B; ++i)
#pragma unroll
            for (int j = 0; j < B; ++j) acc[i] = __fma_rn((double)av[d][i * B + j], xv[d][j], acc[i]);
}

// y = D x of one block.
template <int B, class M>
__device__ __forceinline__ void block_mul(const M (&av)[B * B], const double (&x)[B], double (&y)[B])
{
#pragma unroll
    for (int i = 0; i < B; ++i) {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < B; ++j) s = __fma_rn((double)av[i * B + j], x[j], s);
        y[i] = s;
    }
}

// Aggregation of a level's cells: pairs along the directions whose shift is
// 1.  An aggregate has `g` places for black members: the offsets of all
// paired directions but the first, the first one's follows from the colour.
struct Aggregates {
    int sx = 0, sy = 0, sz = 0, g = 1;
    RbGrid fine, coarse;
};

// Black member s of the aggregate (i, j, k): its cell, or -1 (outside).
__device__ __forceinline__ int black_member(const Aggregates& a, int i, int j, int k, int s)
{
    i <<= a.sx;
    j <<= a.sy;
    k <<= a.sz;
    if (a.sx) {
        if (a.sy) {
            j += s & 1;
            s >>= 1;
        }
        if (a.sz) k += s & 1;
        i += 1 ^ ((i + j + k) & 1);
    } else if (a.sy) {
        if (a.sz) k += s & 1;
        j += 1 ^ ((i + j + k) & 1);
    } else {
        k += 1 ^ ((i + j + k) & 1);
    }
    return i < a.fine.nx && j < a.fine.ny && k < a.fine.nz ? i + a.fine.nx * (j + a.fine.ny * k) : -1;
}

// Where a level's finished rows go: alpha z is added to (add) or stored in
// the black members' z of the finer level.
struct UpView {
    Aggregates agg;
    int add = 0;
    double alpha = 1.0;
    double* w = nullptr;  // null: no finer level
};

template <int B, bool CG>
__device__ __forceinline__ void scatter_up(const UpView& u, const Cell& e, const double (&z)[B])
{
    if (u.w == nullptr) return;
    // at most four members; all are read before the first is written
    int c[4];
    double f[4][B];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        c[s] = s < u.agg.g ? black_member(u.agg, e.i, e.j, e.k, s) : -1;
#pragma unroll
        for (int t = 0; t < B; ++t) f[s][t] = 0.0;
        if (u.add && c[s] >= 0) load_bvec<B, double, CG>(u.w, c[s] >> 1, f[s]);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
#pragma unroll
        for (int t = 0; t < B; ++t) f[s][t] = __fma_rn(u.alpha, z[t], f[s][t]);
        if (c[s] >= 0) store_bvec<B, double>(u.w, c[s] >> 1, f[s]);
    }
}

// ---- the steps ------------------------------------------------------------------
// Loops over the rows of a colour for thread `tid` of `nth`, shared by the
// one-step kernels and the fused coarse cycle (see mg_tail_kernel), so that
// both compute every element alike (operations written out: the compiler
// contracted products and sums differently in the shared-memory cycle).  rr, y: red vectors (rr null: zero), rb,
// z: black ones.

template <int B, int ND, class M, bool CG>
__device__ __forceinline__ void red_row(const RbGrid& g, const Cell& e, int q, const M* U, const double* rr,
                                        const double* z, double (&v)[B])
{
    double acc[B];
#pragma unroll
    for (int t = 0; t < B; ++t) acc[t] = v[t] = 0.0;
    if (rr) load_bvec<B, double, CG>(rr, q, v);
    stencil_dot<B, ND, M, CG>(g, e, q, g.nr, U, z, acc);
#pragma unroll
    for (int t = 0; t < B; ++t) v[t] = __dsub_rn(v[t], acc[t]);
}

// y = rr - U z
template <int B, int ND, class M, bool CG>
__device__ __forceinline__ void rb_y_rows(const RbGrid& g, const RbMatrix<const M>& m, const double* rr,
                                          const double* z, double* y, int tid, int nth)
{
    for (int q = tid; q < g.nr; q += nth) {
        double v[B];
        red_row<B, ND, M, CG>(g, cell_of(g, 0, q), q, m.U, rr, z, v);
        store_bvec<B, double>(y, q, v);
    }
}

// D_r^-1 (rr - U z), handed to the finer level (nothing else reads it).
template <int B, int ND, class M, bool CG>
__device__ __forceinline__ void rb_fin_rows(const RbGrid& g, const RbMatrix<const M>& m, const double* rr,
                                            const double* z, const UpView& up, int tid, int nth)
{
    for (int q = tid; q < g.nr; q += nth) {
        const Cell e = cell_of(g, 0, q);
        M dv[B * B];
        double v[B], x[B];
        load_block<B * B, M>(m.dr + (size_t)q * B * B, dv);
        red_row<B, ND, M, CG>(g, e, q, m.U, rr, z, v);
        block_mul<B, M>(dv, v, x);
        scatter_up<B, CG>(up, e, x);
    }
}

// z = D_b^-1 (rb - L rr): the sweep from z = 0.
template <int B, int ND, class M, bool CG>
__device__ __forceinline__ void rb_pre_rows(const RbGrid& g, const RbMatrix<const M>& m, const double* rr,
                                            const double* rb, double* z, int tid, int nth)
{
    const int nk = g.n - g.nr;
    for (int q = tid; q < nk; q += nth) {
        M dv[B * B];
        double acc[B], v[B], x[B];
#pragma unroll
        for (int t = 0; t < B; ++t) acc[t] = 0.0;
        load_bvec<B, double, CG>(rb, q, v);
        load_block<B * B, M>(m.db + (size_t)q * B * B, dv);
        if (rr) stencil_dot<B, ND, M, CG>(g, cell_of(g, 1, q), q, nk, m.L, rr, acc);
#pragma unroll
        for (int t = 0; t < B; ++t) v[t] = __dsub_rn(v[t], acc[t]);
        block_mul<B, M>(dv, v, x);
        store_bvec<B, double>(z, q, x);
    }
}

// t = rb - A_bb z - L y of one black row.
template <int B, int ND, class M, bool CG>
__device__ __forceinline__ void residual_row(const RbGrid& g, const Cell& e, int q, const RbMatrix<const M>& m,
                                             const double* rb, const double* y, const double (&z)[B], double (&t)[B])
{
    M av[B * B];
    double acc[B], az[B];
#pragma unroll
    for (int c = 0; c < B; ++c) acc[c] = 0.0;
    load_bvec<B, double, CG>(rb, q, t);
    load_block<B * B, M>(m.abb + (size_t)q * B * B, av);
    stencil_dot<B, ND, M, CG>(g, e, q, g.n - g.nr, m.L, y, acc);
    block_mul<B, M>(av, z, az);
#pragma unroll
    for (int c = 0; c < B; ++c) t[c] = __dsub_rn(__dsub_rn(t[c], az[c]), acc[c]);
}

// Coarse right-hand side: the sum of t over the black members of each
// aggregate, g lanes per aggregate in the order of the coarse cells (a
// member's row follows its neighbour's: whole segments), summed by a
// butterfly over the g lanes.  rc: red coarse cells, then black ones.
template <int B, int ND, class M, bool CG>
__device__ __forceinline__ void rb_res_rows(const Aggregates& a, const RbMatrix<const M>& m, const double* rb,
                                            const double* y, const double* z, double* rc, int tid, int nth)
{
    const int items = a.coarse.n * a.g, padded = (items + 31) & ~31, lg = a.g == 4 ? 2 : a.g - 1;
    for (int it = tid; it < padded; it += nth) {
        const Cell C = cell_at(a.coarse, it < items ? it >> lg : 0);
        const int c = it < items ? black_member(a, C.i, C.j, C.k, it & (a.g - 1)) : -1;
        double t[B];
#pragma unroll
        for (int v = 0; v < B; ++v) t[v] = 0.0;
        if (c >= 0) {
            const int q = c >> 1;
            double zv[B];
            load_bvec<B, double, CG>(z, q, zv);
            residual_row<B, ND, M, CG>(a.fine, cell_at(a.fine, c), q, m, rb, y, zv, t);
        }
        for (int o = 1; o < a.g; o <<= 1)
#pragma unroll
            for (int v = 0; v < B; ++v) t[v] += __shfl_xor_sync(0xffffffffu, t[v], o);
        if (it < items && (it & (a.g - 1)) == 0)
            store_bvec<B, double>(rc, (C.c >> 1) + (((C.i + C.j + C.k) & 1) ? a.coarse.nr : 0), t);
    }
}

// The same of the right-hand side itself (rr null: zero), for a level
// without pre-smoothing: pairs, a black member and the red one beside it.
template <int B, bool CG>
__device__ __forceinline__ void rb_restrict_rows(const Aggregates& a, const double* rr, const double* rb, double* rc,
                                                 int tid, int nth)
{
    for (int p = tid; p < a.coarse.n; p += nth) {
        const Cell C = cell_at(a.coarse, p);
        double s[B];
#pragma unroll
        for (int t = 0; t < B; ++t) s[t] = 0.0;
        const int i0 = C.i << a.sx, j0 = C.j << a.sy, k0 = C.k << a.sz;
        for (int o = 0; o < (1 << (a.sx + a.sy + a.sz)); ++o) {
            const int i = i0 + (a.sx ? o & 1 : 0), j = j0 + (a.sy ? (o >> a.sx) & 1 : 0), k = k0 + (a.sz ? o >> (a.sx + a.sy) : 0);
            if (i >= a.fine.nx || j >= a.fine.ny || k >= a.fine.nz) continue;
            const double* r = ((i + j + k) & 1) ? rb : rr;
            if (!r) continue;
            double v[B];
            load_bvec<B, double, CG>(r, (i + a.fine.nx * (j + a.fine.ny * k)) >> 1, v);
#pragma unroll
            for (int t = 0; t < B; ++t) s[t] += v[t];
        }
        store_bvec<B, double>(rc, (p >> 1) + (((C.i + C.j + C.k) & 1) ? a.coarse.nr : 0), s);
    }
}

// z += D_b^-1 (rb - A_bb z - L y), handed to the finer level.
template <int B, int ND, class M, bool CG>
__device__ __forceinline__ void rb_post_rows(const RbGrid& g, const RbMatrix<const M>& m, const double* rb,
                                             const double* y, double* z, const UpView& up, int tid, int nth)
{
    const int nk = g.n - g.nr;
    for (int q = tid; q < nk; q += nth) {
        const Cell e = cell_of(g, 1, q);
        M dv[B * B];
        double zv[B], t[B], x[B];
        load_bvec<B, double, CG>(z, q, zv);
        load_block<B * B, M>(m.db + (size_t)q * B * B, dv);
        residual_row<B, ND, M, CG>(g, e, q, m, rb, y, zv, t);
        block_mul<B, M>(dv, t, x);
#pragma unroll
        for (int c = 0; c < B; ++c) zv[c] = __dadd_rn(zv[c], x[c]);
        store_bvec<B, double>(z, q, zv);
        scatter_up<B, CG>(up, e, zv);
    }
}

// The coarsest level: inv r, a warp per unknown (see dense_rows; red cells,
// then black ones), handed to the finer level.
template <int B, class M, bool CG>
__device__ __forceinline__ void rb_dense_rows(const RbGrid& g, const M* __restrict__ inv, const double* r,
                                              const UpView& up, int tid, int nth)
{
    const int lane = tid & 31, n = g.n * B;
    for (int i = tid >> 5; i < n; i += nth >> 5) {
        double s = 0.0;
        for (int j = lane; j < n; j += 32) s = __fma_rn((double)inv[i * n + j], CG ? __ldcg(r + j) : r[j], s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const int P = i / B, c = i - P * B;
        if (lane < up.agg.g) {
            const Cell e = P < g.nr ? cell_of(g, 0, P) : cell_of(g, 1, P - g.nr);
            const int f = black_member(up.agg, e.i, e.j, e.k, lane);
            if (f >= 0) {
                double* w = up.w + (size_t)(f >> 1) * B + c;
                *w = __fma_rn(up.alpha, s, up.add ? (CG ? __ldcg(w) : *w) : 0.0);
            }
        }
    }
}

// ---- one step per launch ------------------------------------------------------
template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_y_kernel(RbGrid g, RbMatrix<const M> m, const double* rr, const double* z,
                                                   double* y, const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_y_rows<B, ND, M, false>(g, m, rr, z, y, tid, nth);
}

template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_fin_kernel(RbGrid g, RbMatrix<const M> m, const double* rr, const double* z,
                                                     UpView up, const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_fin_rows<B, ND, M, false>(g, m, rr, z, up, tid, nth);
}

template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_pre_kernel(RbGrid g, RbMatrix<const M> m, const double* rr, const double* rb,
                                                     double* z, const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_pre_rows<B, ND, M, false>(g, m, rr, rb, z, tid, nth);
}

template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_res_kernel(Aggregates a, RbMatrix<const M> m, const double* rb,
                                                     const double* y, const double* z, double* rc, const KScal* sc,
                                                     int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_res_rows<B, ND, M, false>(a, m, rb, y, z, rc, tid, nth);
}

template <int B>
__global__ void __launch_bounds__(512, 1) rb_restrict_kernel(Aggregates a, const double* rr, const double* rb, double* rc,
                                                          const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_restrict_rows<B, false>(a, rr, rb, rc, tid, nth);
}

template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_post_kernel(RbGrid g, RbMatrix<const M> m, const double* rb, const double* y,
                                                      double* z, UpView up, const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    THREAD_RANGE;
    rb_post_rows<B, ND, M, false>(g, m, rb, y, z, up, tid, nth);
}

template <int B, class M>
__global__ void __launch_bounds__(1024) rb_dense_kernel(RbGrid g, const M* __restrict__ inv, const double* r, UpView up,
                                                        const KScal* sc, int skip_if_s)
{
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    rb_dense_rows<B, M, false>(g, inv, r, up, (int)threadIdx.x, (int)blockDim.x);
}

// ---- BiCGStab on the black half ------------------------------------------------
// b (red cells, then black ones) from the natural order, component after
// component.
template <int B>
__global__ void rb_permute_kernel(RbGrid g, const double* __restrict__ rhs, double* __restrict__ b)
{
    GRID_STRIDE(c64, g.n)
    {
        const Cell e = cell_at(g, (int)c64);
        const int P = (e.c >> 1) + (((e.i + e.j + e.k) & 1) ? g.nr : 0);
        double v[B];
#pragma unroll
        for (int t = 0; t < B; ++t) v[t] = rhs[(size_t)t * g.n + e.c];
        store_bvec<B, double>(b, P, v);
    }
}

// b_b - L b_r is the first residual; with the vectors' start values, the
// shadow residual, and the dots of bicg_init (rr of the residual, thr of the
// whole b).
template <int B, int ND>
__global__ void __launch_bounds__(kThreads) rb_init_kernel(RbGrid g, RbMatrix<const double> m,
                                                           const double* __restrict__ b, double* r, double* rhat,
                                                           double* p, double* v, double* x, double* partials,
                                                           unsigned int* counter, KScal* sc, double tol2)
{
    const int nk = g.n - g.nr;
    const double* bb = b + (size_t)g.nr * B;
    double d[3] = {0.0, 0.0, 0.0};
    GRID_STRIDE(i64, g.nr)
    {
        const int q = (int)i64;
        double w[B];
        load_bvec<B, double>(b, q, w);
#pragma unroll
        for (int t = 0; t < B; ++t) d[2] += w[t] * w[t];
        if (q >= nk) continue;
        double acc[B];
#pragma unroll
        for (int t = 0; t < B; ++t) acc[t] = 0.0;
        stencil_dot<B, ND, double, false>(g, cell_of(g, 1, q), q, nk, m.L, b, acc);
        load_bvec<B, double>(bb, q, w);
#pragma unroll
        for (int t = 0; t < B; ++t) {
            const int64_t i = (int64_t)q * B + t;
            const double gi = w[t] - acc[t], hi = shadow_entry(i);
            d[2] += w[t] * w[t];
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

// v = S z = A_bb z + L y (y = -U z), with the dots of bicg_spmv_alpha (OMEGA
// false: alpha = rho_new / (h . v), h the shadow residual) or
// bicg_spmv_omega (omega = (v . h) / (v . v), h = s).
template <int B, int ND, bool OMEGA>
__global__ void __launch_bounds__(kThreads, 2)
    rb_spmv_kernel(RbGrid g, RbMatrix<const double> m, const double* __restrict__ z, const double* __restrict__ y,
                   const double* __restrict__ h, double* __restrict__ v, double* partials, unsigned int* counter,
                   KScal* sc)
{
    pdl_wait();
    if (stopped(sc) || (OMEGA && sc->s_conv)) return;
    constexpr int ND_ = OMEGA ? 2 : 1;
    const int nk = g.n - g.nr;
    double d[ND_];
#pragma unroll
    for (int k = 0; k < ND_; ++k) d[k] = 0.0;
    GRID_STRIDE(q64, nk)
    {
        const int q = (int)q64;
        double acc[B], zv[B], az[B], hv[B];
#pragma unroll
        for (int t = 0; t < B; ++t) acc[t] = 0.0;
        double av[B * B];
        load_bvec<B, double>(z, q, zv);
        load_bvec<B, double>(h, q, hv);
        load_block<B * B, double>(m.abb + (size_t)q * B * B, av);
        stencil_dot<B, ND, double, false>(g, cell_of(g, 1, q), q, nk, m.L, y, acc);
        block_mul<B, double>(av, zv, az);
#pragma unroll
        for (int t = 0; t < B; ++t) acc[t] += az[t];
        store_bvec<B, double>(v, q, acc);
#pragma unroll
        for (int t = 0; t < B; ++t) {
            d[0] += hv[t] * acc[t];
            if (OMEGA) d[ND_ - 1] += acc[t] * acc[t];
        }
    }
    double s[ND_];
    if (grid_sum<ND_>(d, partials, counter, s)) {
        if (OMEGA) {
            sc->ts = s[0];
            sc->tt = s[ND_ - 1];
            if (s[ND_ - 1] == 0.0 || !isfinite(s[ND_ - 1])) sc->status = ST_BREAK;
            else sc->omega = s[0] / s[ND_ - 1];
        } else {
            sc->rv = s[0];
            if (s[0] == 0.0 || !isfinite(s[0])) sc->status = ST_BREAK;
            else sc->alpha = sc->rho_new / s[0];
        }
    }
}

// The solution in the natural order: x_b, and x_r = D_r^-1 (b_r - U x_b).
template <int B, int ND>
__global__ void __launch_bounds__(kThreads) rb_solution_kernel(RbGrid g, RbMatrix<const double> m,
                                                               const double* __restrict__ b,
                                                               const double* __restrict__ x, double* __restrict__ out)
{
    const int nk = g.n - g.nr;
    GRID_STRIDE(q64, g.nr)
    {
        const int q = (int)q64;
        const Cell e = cell_of(g, 0, q);
        double v[B], z[B];
        double dv[B * B];
        load_block<B * B, double>(m.dr + (size_t)q * B * B, dv);
        red_row<B, ND, double, false>(g, e, q, m.U, b, x, v);
        block_mul<B, double>(dv, v, z);
#pragma unroll
        for (int t = 0; t < B; ++t) out[(size_t)t * g.n + e.c] = z[t];
        if (q >= nk) continue;
        const Cell f = cell_of(g, 1, q);
        load_bvec<B, double>(x, q, z);
#pragma unroll
        for (int t = 0; t < B; ++t) out[(size_t)t * g.n + f.c] = z[t];
    }
}

// ---- set-up ---------------------------------------------------------------------
// Where the Jacobian's entries go, one thread per row (component after
// component): map[position in A] = entry.  bad |= 1: an entry that couples
// cells which are no neighbours; 2: a row without its diagonal entry.
__global__ void rb_map_kernel(RbGrid g, int B, int nd, const int* __restrict__ rowptr, const int* __restrict__ colind,
                              int* __restrict__ map, int* bad)
{
    const int nk = g.n - g.nr, bb = B * B;
    int flags = 0;
    GRID_STRIDE(u, (int64_t)g.n * B)
    {
        const int cu = (int)(u / g.n);
        const Cell e = cell_at(g, (int)(u - (int64_t)cu * g.n));
        const int colour = (e.i + e.j + e.k) & 1, q = e.c >> 1, rows = colour ? nk : g.nr;
        const size_t off = colour ? (size_t)nd * g.nr : 0, dia = (size_t)nd * g.n + (colour ? g.nr : 0);
        bool has = false;
        for (int t = rowptr[u]; t < rowptr[u + 1]; ++t) {
            const int col = colind[t], cv = col / g.n, c = col - cv * g.n, diff = c - e.c;
            size_t slot;
            if (diff == 0) {
                slot = dia + q;
                has = has || cv == cu;
            } else {
                // the direction whose neighbour c is (sides of 1 make two
                // offsets equal: the one that exists)
                int d = 0, nq = 0;
                for (; d < nd; ++d) {
                    const int o = d < 2 ? 1 : d < 4 ? g.nx : g.step;
                    if (diff == (d & 1 ? o : -o) && neighbour(g, e, d, nq)) break;
                }
                if (d == nd) {
                    flags |= 1;
                    continue;
                }
                slot = off + (size_t)d * rows + q;
            }
            map[slot * bb + cu * B + cv] = t;
        }
        if (!has) flags |= 2;
    }
    if (flags) atomicOr(bad, flags);
}

// A from the Jacobian's values.  A tile of 32 cells of a colour takes all its
// directions in turn, so that the sectors of its Jacobian rows, read eight
// bytes at a time, are read again from L1.
__global__ void __launch_bounds__(kThreads) rb_gather_kernel(RbGrid g, int bb, int nd, const int* __restrict__ map,
                                                             const double* __restrict__ j, double* __restrict__ a)
{
    const int nk = g.n - g.nr;
    const int red_tiles = (g.nr + 31) / 32, tiles = red_tiles + (nk + 31) / 32;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const bool red = tile < red_tiles;
        const int rows = red ? g.nr : nk, q0 = (red ? tile : tile - red_tiles) * 32;
        const int w = min(32, rows - q0) * bb;
        for (int x = threadIdx.x; x < w * (nd + 1); x += blockDim.x) {
            const int d = x / w;
            const size_t row = d < nd ? (red ? 0 : (size_t)nd * g.nr) + (size_t)d * rows : (size_t)nd * g.n + (red ? 0 : g.nr);
            const size_t p = (row + q0) * bb + (x - d * w);
            const int e = map[p];
            a[p] = e >= 0 ? j[e] : 0.0;
        }
    }
}

// Mean share that each direction has of a cell's couplings of a component
// with itself, weighted by how strongly the row is coupled at all (shares of
// its diagonal entry, at most 1).
__global__ void __launch_bounds__(kThreads) rb_strength_kernel(RbGrid g, int B, int nd, const double* __restrict__ a,
                                                               double* partials, unsigned int* counter, double* out)
{
    const int bb = B * B;
    const RbMatrix<const double> m(a, nd, bb, g.n, g.nr);
    double sum[3] = {0.0, 0.0, 0.0};
    GRID_STRIDE(P64, g.n)
    {
        const int P = (int)P64;
        const bool red = P < g.nr;
        const int rows = red ? g.nr : g.n - g.nr, q = red ? P : P - g.nr;
        for (int c = 0; c < B; ++c) {
            const int e = c * B + c;
            const double diag = fabs((red ? m.dr : m.abb)[(size_t)q * bb + e]);
            double s[3] = {0.0, 0.0, 0.0};
            for (int d = 0; d < nd; ++d) s[d >> 1] += fabs((red ? m.U : m.L)[((size_t)d * rows + q) * bb + e]);
            const double all = s[0] + s[1] + s[2];
            if (!(all > 0.0) || !(diag > 0.0) || !isfinite(all / diag)) continue;
            const double w = fmin(1.0, all / diag) / all;
            for (int t = 0; t < 3; ++t) sum[t] += w * s[t];
        }
    }
    double s[3];
    if (grid_sum<3>(sum, partials, counter, s))
        for (int t = 0; t < 3; ++t) out[t] = s[t];
}

// The coarse matrix R A R^T of a 0/1 aggregation, one thread per value of a
// coarse cell: the blocks of its members that cross each of its faces, and
// its diagonal block with the couplings inside it, summed in the order of
// the members and directions.
__global__ void __launch_bounds__(kThreads) rb_galerkin_kernel(Aggregates a, int bb, int nd, const double* __restrict__ fa,
                                                               double* __restrict__ ca)
{
    const RbGrid &f = a.fine, &g = a.coarse;
    const RbMatrix<const double> F(fa, nd, bb, f.n, f.nr);
    const RbMatrix<double> G(ca, nd, bb, g.n, g.nr);
    GRID_STRIDE(x, (int64_t)g.n * bb)
    {
        const int c = (int)(x / bb), e = (int)(x - (int64_t)c * bb);
        const Cell C = cell_at(g, c);
        const bool red = ((C.i + C.j + C.k) & 1) == 0;
        const int q = c >> 1, rows = red ? g.nr : g.n - g.nr;
        double diag = 0.0, off[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int o = 0; o < 8; ++o) {
            const int dx = o & 1, dy = (o >> 1) & 1, dz = o >> 2;
            if ((dx && !a.sx) || (dy && !a.sy) || (dz && !a.sz)) continue;
            Cell m;
            m.i = (C.i << a.sx) + dx;
            m.j = (C.j << a.sy) + dy;
            m.k = (C.k << a.sz) + dz;
            if (m.i >= f.nx || m.j >= f.ny || m.k >= f.nz) continue;
            m.c = m.i + f.nx * (m.j + f.ny * m.k);
            const bool mr = ((m.i + m.j + m.k) & 1) == 0;
            const int mq = m.c >> 1, mrows = mr ? f.nr : f.n - f.nr;
            diag += (mr ? F.dr : F.abb)[(size_t)mq * bb + e];
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                if (d >= nd) break;
                int nq;
                if (!neighbour(f, m, d, nq)) continue;
                const double v = (mr ? F.U : F.L)[((size_t)d * mrows + mq) * bb + e];
                // inside the aggregate: the direction is paired and leads to
                // the other half
                const bool inner = d < 2 ? a.sx && dx != (d & 1) : d < 4 ? a.sy && dy != (d & 1) : a.sz && dz != (d & 1);
                if (inner) diag += v;
                else off[d] += v;
            }
        }
        (red ? G.dr : G.abb)[(size_t)q * bb + e] = diag;
#pragma unroll
        for (int d = 0; d < 6; ++d)
            if (d < nd) (red ? G.U : G.L)[((size_t)d * rows + q) * bb + e] = off[d];
    }
}

// D_r^-1 over the red cells.
template <int B>
__global__ void __launch_bounds__(kThreads) rb_factor_red_kernel(RbGrid g, double* __restrict__ dr, int* status)
{
    constexpr int BB = B * B;
    GRID_STRIDE(q, g.nr)
    {
        double d[BB];
#pragma unroll
        for (int e = 0; e < BB; ++e) d[e] = dr[q * BB + e];
        if (!invert_block<B>(d)) *status = 1;
#pragma unroll
        for (int e = 0; e < BB; ++e) dr[q * BB + e] = d[e];
    }
}

// L = A_br D_r^-1 and D_b^-1 = (A_bb - sum L U)^-1 over the black cells: of
// L U only the diagonal block is in the pattern (block ILU(0)).
template <int B, int ND>
__global__ void __launch_bounds__(kThreads) rb_factor_black_kernel(RbGrid g, RbMatrix<double> m, int* status)
{
    constexpr int BB = B * B;
    const int nk = g.n - g.nr;
    GRID_STRIDE(q64, nk)
    {
        const int q = (int)q64;
        const Cell e = cell_of(g, 1, q);
        double D[BB];
#pragma unroll
        for (int t = 0; t < BB; ++t) D[t] = m.abb[(size_t)q * BB + t];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            int nq;
            if (!neighbour(g, e, d, nq)) continue;
            double* lp = m.L + ((size_t)d * nk + q) * BB;
            const double* up = m.U + ((size_t)(d ^ 1) * g.nr + nq) * BB;  // the red cell's block towards this one
            const double* dp = m.dr + (size_t)nq * BB;
            double av[BB], dv[BB], uv[BB], l[BB];
            load_block<BB, double>(lp, av);
            load_block<BB, double>(dp, dv);
            load_block<BB, double>(up, uv);
#pragma unroll
            for (int i = 0; i < B; ++i)
#pragma unroll
                for (int j = 0; j < B; ++j) {
                    double s = 0.0;
#pragma unroll
                    for (int t = 0; t < B; ++t) s += av[i * B + t] * dv[t * B + j];
                    l[i * B + j] = s;
                }
#pragma unroll
            for (int i = 0; i < B; ++i)
#pragma unroll
                for (int j = 0; j < B; ++j) {
                    double s = 0.0;
#pragma unroll
                    for (int t = 0; t < B; ++t) s += l[i * B + t] * uv[t * B + j];
                    D[i * B + j] -= s;
                }
#pragma unroll
            for (int t = 0; t < BB; ++t) lp[t] = l[t];
        }
        if (!invert_block<B>(D)) *status = 1;
#pragma unroll
        for (int t = 0; t < BB; ++t) m.db[(size_t)q * BB + t] = D[t];
    }
}

// The coarsest matrix, dense and row-major (red cells, then black ones), for
// dense_inverse_kernel; `dense` is zero beforehand.
__global__ void rb_dense_fill_kernel(RbGrid g, int B, int nd, const double* __restrict__ a, double* __restrict__ dense)
{
    const int bb = B * B, n = g.n * B;
    const RbMatrix<const double> m(a, nd, bb, g.n, g.nr);
    GRID_STRIDE(P64, g.n)
    {
        const int P = (int)P64;
        const bool red = P < g.nr;
        const int rows = red ? g.nr : g.n - g.nr, q = red ? P : P - g.nr;
        const Cell e = cell_of(g, red ? 0 : 1, q);
        for (int t = 0; t < bb; ++t)
            dense[(size_t)(P * B + t / B) * n + P * B + t % B] = (red ? m.dr : m.abb)[(size_t)q * bb + t];
        for (int d = 0; d < nd; ++d) {
            int nq;
            if (!neighbour(g, e, d, nq)) continue;
            const int Q = red ? g.nr + nq : nq;
            for (int t = 0; t < bb; ++t)
                dense[(size_t)(P * B + t / B) * n + Q * B + t % B] = (red ? m.U : m.L)[((size_t)d * rows + q) * bb + t];
        }
    }
}

// ---- the coarse end of the cycle in one kernel ----------------------------------
// As mg_tail_kernel: one thread-block cluster, a cluster barrier between the
// steps, the coarsest levels in block 0's shared memory.
template <class M>
struct RbTailLevel {
    RbGrid g;
    int coarsest = 0, pre = 1;
    const M* a = nullptr;           // matrix (RbMatrix), or the dense inverse of the coarsest level
    const double* rr = nullptr;     // right-hand side, red (null: zero) and black
    const double* rb = nullptr;
    double* r = nullptr;            // where the finer level's restriction writes it
    double* z = nullptr;            // black iterate
    double* y = nullptr;            // red work vector
    Aggregates agg;                 // to the next level
    UpView up;                      // where its rows go
    int so_a = 0, so_r = 0, so_w = 0;  // offsets in block 0's shared memory
};

template <class M>
struct RbTailParams {
    RbTailLevel<M> lv[kMaxTail];
    int nlev = 0;
    int local_first = kMaxTail;
    int nregions = 0;
    int ncopies = 0;
    PrefetchRegion reg[kMaxTail];
    TailCopy copies[kMaxTail];
    long long* trace = nullptr;
};
static_assert(sizeof(RbTailParams<double>) <= 4096, "fused cycle parameters exceed 4 KB");

// One level's steps down to the coarse right-hand side rc; sync() ends a step.
template <int B, int ND, class M, bool CG, class Sync>
__device__ __forceinline__ void rb_down(const RbTailLevel<M>& L, const RbMatrix<const M>& m, const double* rr,
                                        const double* rb, double* z, double* y, double* rc, int tid, int nth,
                                        Sync&& sync)
{
    if (L.pre) {
        rb_pre_rows<B, ND, M, CG>(L.g, m, rr, rb, z, tid, nth);
        sync();
        rb_y_rows<B, ND, M, CG>(L.g, m, rr, z, y, tid, nth);
        sync();
        rb_res_rows<B, ND, M, CG>(L.agg, m, rb, y, z, rc, tid, nth);
    } else {
        rb_restrict_rows<B, CG>(L.agg, rr, rb, rc, tid, nth);
    }
    sync();
}

template <int B, int ND, class M, bool CG, class Sync>
__device__ __forceinline__ void rb_up(const RbTailLevel<M>& L, const RbMatrix<const M>& m, const double* rr,
                                      const double* rb, double* z, double* y, const UpView& up, int tid, int nth,
                                      Sync&& sync)
{
    rb_y_rows<B, ND, M, CG>(L.g, m, rr, z, y, tid, nth);
    sync();
    rb_post_rows<B, ND, M, CG>(L.g, m, rb, y, z, up, tid, nth);
    if (up.w == nullptr) return;
    sync();
    rb_fin_rows<B, ND, M, CG>(L.g, m, rr, z, up, tid, nth);
    sync();
}

// The levels from lf on, on block 0 alone, in its shared memory; the
// correction goes to level lf - 1's z in global memory.
template <int B, int ND, class M>
__device__ void rb_local_cycle(const RbTailParams<M>& p, int lf, unsigned char* sm)
{
    const int tid = (int)threadIdx.x, nth = (int)blockDim.x;
    auto sync = [] { __syncthreads(); };
    auto at_r = [&](int l) { return (double*)(sm + p.lv[l].so_r); };
    auto at_y = [&](int l) { return (double*)(sm + p.lv[l].so_w); };
    auto at_z = [&](int l) { return at_y(l) + p.lv[l].g.nr * B; };
    auto matrix = [&](int l) {
        const RbGrid& g = p.lv[l].g;
        return RbMatrix<const M>((const M*)(sm + p.lv[l].so_a), ND, B * B, g.n, g.nr);
    };
    auto up_of = [&](int l) {
        UpView u = p.lv[l].up;
        if (l > lf) u.w = at_z(l - 1);
        return u;
    };
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (int i = tid; i < p.lv[lf].g.n * B; i += nth) at_r(lf)[i] = __ldcg(p.lv[lf].rr + i);
    __syncthreads();
    int l = lf;
    for (; !p.lv[l].coarsest; ++l)
        rb_down<B, ND, M, false>(p.lv[l], matrix(l), at_r(l), at_r(l) + p.lv[l].g.nr * B, at_z(l), at_y(l),
                                 at_r(l + 1), tid, nth, sync);
    rb_dense_rows<B, M, false>(p.lv[l].g, (const M*)(sm + p.lv[l].so_a), at_r(l), up_of(l), tid, nth);
    __syncthreads();
    for (--l; l >= lf; --l)
        rb_up<B, ND, M, false>(p.lv[l], matrix(l), at_r(l), at_r(l) + p.lv[l].g.nr * B, at_z(l), at_y(l), up_of(l),
                               tid, nth, sync);
}

template <int B, int ND, class M>
__global__ void __launch_bounds__(kTailThreads, 1)
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
    // 32 rows (a warp) at a time, round robin over the blocks
    const int tid = (((int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x) << 5) | (int)(threadIdx.x & 31);
    const int nth = (int)(gridDim.x * blockDim.x);
    auto matrix = [&](const RbTailLevel<M>& L) { return RbMatrix<const M>(L.a, ND, B * B, L.g.n, L.g.nr); };
    int l = 0;
    for (; l < lf && !p.lv[l].coarsest; ++l) {
        const RbTailLevel<M>& L = p.lv[l];
        rb_down<B, ND, M, true>(L, matrix(L), L.rr, L.rb, L.z, L.y, p.lv[l + 1].r, tid, nth, sync);
    }
    if (l == lf) {
        // block 0 alone; the other blocks wait at the next cluster barrier
        if (blockIdx.x == 0) rb_local_cycle<B, ND, M>(p, lf, tail_smem);
    } else {
        rb_dense_rows<B, M, true>(p.lv[l].g, p.lv[l].a, p.lv[l].rr, p.lv[l].up, tid, nth);
    }
    sync();
    for (--l; l >= 0; --l) {
        const RbTailLevel<M>& L = p.lv[l];
        rb_up<B, ND, M, true>(L, matrix(L), L.rr, L.rb, L.z, L.y, L.up, tid, nth, sync);
    }
}
