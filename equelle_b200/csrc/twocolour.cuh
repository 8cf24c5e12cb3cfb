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
//   y   = r_r - U z_b                       (rb_y_kernel)
//   t_b = r_b - A_bb z_b - L y              (the residual; red rows: 0)
//   z_b += D_b^-1 t_b                       (rb_post_kernel)
//   z_r = D_r^-1 (r_r - U z_b)              (rb_fin_kernel)
// is one sweep from any z_b: the red part of the iterate is never needed
// before the last line, the residual of the down-leg is summed straight into
// the coarse right-hand side (rb_res_kernel), and the coarse level's last two
// steps add alpha times their rows to the fine black cells (UpRow).  A
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
// dependent steps on the coarse ones.  Krylov time of one time step in the
// general form with 2 x 2 x 2 aggregates and in this one: two-phase 128x128x64
// 150 ms (203 iterations) and 44 (90), 512x512 26.5 and 8.9, 33x31x17 20.6 and
// 6.2, impes 97x83x41 31.6 and 8.6.  First step of a new 128x128x64 runtime,
// with the analysis on the host and on the device: 756 and 154 ms.

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

// One block of a level's matrix, which no kernel of a solve writes: read past
// L1 (every block is used once per kernel; 3 x 3 blocks through it, since the
// lanes' single values share sectors), and where it stands relative to pdl_wait
// (the assembly statements keep their order).
template <int BB, class M>
__device__ __forceinline__ void load_matrix(const M* p, M (&v)[BB])
{
    if constexpr (BB == 4 && sizeof(M) == 8) {
        asm volatile("ld.global.nc.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
    } else if constexpr (BB == 4) {
        asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
    } else if constexpr (BB == 9 && sizeof(M) == 8) {
#pragma unroll
        for (int e = 0; e < BB; ++e) asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v[e]) : "l"(p + e));
    } else if constexpr (BB == 9) {
#pragma unroll
        for (int e = 0; e < BB; ++e) asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v[e]) : "l"(p + e));
    } else if constexpr (sizeof(M) == 8) {
#pragma unroll
        for (int e = 0; e < BB; ++e) asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v[e]) : "l"(p + e));
    } else {
#pragma unroll
        for (int e = 0; e < BB; ++e) asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v[e]) : "l"(p + e));
    }
}

// A row's off-diagonal blocks and its neighbours' numbers.  load() reads
// nothing that a solve writes; dot() adds sum A_d x_d to acc, directions in
// order.  The loads are unconditional, so that all of them are issued before
// the first sum (with a branch per neighbour the compiler waited for each one
// in turn, in 34 registers): the block of a missing neighbour is stored as
// zero, and the vector is then read at the row's own number, or the last one.
//
// A row of 3 x 3 FP64 blocks is more than fits in registers beside them (rows of
// six spilled 84 to 780 bytes): half of it comes ahead, the other half after
// the first half's sums.  With that, and 3 x 3 blocks through L1: an iteration
// of three species on 96^3 cells 1515 -> 963 us (general form 1335), 64^3 580 ->
// 417, 600x600 580 -> 440.
template <int B, int ND, class M>
struct StencilRow {
    static constexpr int G = B * B * ND * (int)sizeof(M) > 256 ? ND / 2 : ND;  // directions ahead
    M av[G][B * B];
    int nq[ND];
    const M* rest;  // the blocks of direction G
    int stride;     // rows of the colour
    // row q of `rows`, cell e
    __device__ __forceinline__ void load(const RbGrid& g, const Cell& e, int q, int rows, const M* a)
    {
        const int own = max(min(q, g.n - rows - 1), 0);  // the other colour has n - rows cells
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            if (!neighbour(g, e, d, nq[d])) nq[d] = own;
            if (d < G) load_matrix<B * B, M>(a + ((size_t)d * rows + q) * (B * B), av[d]);
        }
        rest = a + ((size_t)G * rows + q) * (B * B);
        stride = rows;
    }
    __device__ __forceinline__ void dot(const double* x, double (&acc)[B]) const
    {
        sums(0, av, x, acc);
        if constexpr (G < ND) {
            M bv[ND - G][B * B];
#pragma unroll
            for (int d = G; d < ND; ++d) load_matrix<B * B, M>(rest + (size_t)(d - G) * stride * (B * B), bv[d - G]);
            sums(G, bv, x, acc);
        }
    }

private:
    template <int N>
    __device__ __forceinline__ void sums(int d0, const M (&v)[N][B * B], const double* x, double (&acc)[B]) const
    {
        double xv[N][B];
#pragma unroll
        for (int d = 0; d < N; ++d) load_bvec<B, double>(x, nq[d0 + d], xv[d]);
#pragma unroll
        for (int d = 0; d < N; ++d)
#pragma unroll
            for (int i = 0; i < B; ++i)
#pragma unroll
                for (int j = 0; j < B; ++j) acc[i] = __fma_rn((double)v[d][i * B + j], xv[d][j], acc[i]);
    }
};

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

// The fine members of one row (at most four) and their values, read before
// the row is computed.
template <int B>
struct UpRow {
    int c[4];
    double f[4][B];
    __device__ __forceinline__ void members(const UpView& u, const Cell& e)
    {
#pragma unroll
        for (int s = 0; s < 4; ++s)
            c[s] = u.w != nullptr && s < u.agg.g ? black_member(u.agg, e.i, e.j, e.k, s) : -1;
    }
    template <bool CG = false>
    __device__ __forceinline__ void load(const UpView& u)
    {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
#pragma unroll
            for (int t = 0; t < B; ++t) f[s][t] = 0.0;
            if (u.add && c[s] >= 0) load_bvec<B, double, CG>(u.w, c[s] >> 1, f[s]);
        }
    }
    __device__ __forceinline__ void store(const UpView& u, const double (&z)[B])
    {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
#pragma unroll
            for (int t = 0; t < B; ++t) f[s][t] = __fma_rn(u.alpha, z[t], f[s][t]);
            if (c[s] >= 0) store_bvec<B, double>(u.w, c[s] >> 1, f[s]);
        }
    }
};

// ---- the steps ------------------------------------------------------------------
// One kernel per step.  The resident coarse cycle below computes every
// element alike (operations written out: the compiler contracted products and
// sums differently there).  rr, y: red vectors (rr null: zero), rb, z: black
// ones.

// Rows tid, tid + nth, ... of `rows`: load(q) reads what no kernel of the
// solve writes (matrix blocks, neighbours' numbers), run(q) the rest.  The
// kernel after this one may start as soon as every block here has, and the
// first row's load comes before the wait for the kernel ahead: a step's
// matrix, most of its bytes, comes in while the step before it ends, on SMs
// that this one does not need or has left.  The matrices were complete before
// the solve's first kernel, which is launched without that liberty.  Krylov
// iterations of a step, without and with it: two-phase 48x40 2.77 -> 2.49 ms,
// 255x257 mixed 6.4 -> 5.8, 512x512 10.4 -> 8.9, 33x31x17 7.0 -> 6.2,
// 128x128x64 45.2 -> 43.8 (its finest level takes seven waves of blocks, of
// which only the first gains).  False: nothing ran.
template <class Load, class Run>
__device__ __forceinline__ bool for_rows(int rows, const KScal* sc, int skip_if_s, Load&& load, Run&& run)
{
    pdl_trigger();
    const int tid = (int)(blockIdx.x * blockDim.x + threadIdx.x), nth = (int)(gridDim.x * blockDim.x);
    if (tid < rows) load(tid);
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return false;
    for (int q = tid; q < rows; q += nth) {
        if (q != tid) load(q);
        run(q);
    }
    return true;
}

// v = rr - U z of red row q.
template <int B, int ND, class M>
__device__ __forceinline__ void red_row(const StencilRow<B, ND, M>& row, int q, const double* rr, const double* z,
                                        double (&v)[B])
{
    double acc[B];
#pragma unroll
    for (int t = 0; t < B; ++t) acc[t] = v[t] = 0.0;
    if (rr) load_bvec<B, double>(rr, q, v);
    row.dot(z, acc);
#pragma unroll
    for (int t = 0; t < B; ++t) v[t] = __dsub_rn(v[t], acc[t]);
}

// t = rb - A_bb z - L y of one black row: the blocks of L in row, A_bb in av.
template <int B, int ND, class M>
__device__ __forceinline__ void residual_row(const StencilRow<B, ND, M>& row, const M (&av)[B * B], int q,
                                             const double* rb, const double* y, const double (&z)[B], double (&t)[B])
{
    double acc[B], az[B];
#pragma unroll
    for (int c = 0; c < B; ++c) acc[c] = 0.0;
    load_bvec<B, double>(rb, q, t);
    row.dot(y, acc);
    block_mul<B, M>(av, z, az);
#pragma unroll
    for (int c = 0; c < B; ++c) t[c] = __dsub_rn(__dsub_rn(t[c], az[c]), acc[c]);
}

// y = rr - U z
template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_y_kernel(RbGrid g, RbMatrix<const M> m, const double* rr, const double* z,
                                                   double* y, const KScal* sc, int skip_if_s)
{
    StencilRow<B, ND, M> row;
    for_rows(
        g.nr, sc, skip_if_s, [&](int q) { row.load(g, cell_of(g, 0, q), q, g.nr, m.U); },
        [&](int q) {
            double v[B];
            red_row<B, ND, M>(row, q, rr, z, v);
            store_bvec<B, double>(y, q, v);
        });
}

// D_r^-1 (rr - U z), handed to the finer level (nothing else reads it).
template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_fin_kernel(RbGrid g, RbMatrix<const M> m, const double* rr, const double* z,
                                                     UpView up, const KScal* sc, int skip_if_s)
{
    StencilRow<B, ND, M> row;
    UpRow<B> fine;
    M dv[B * B];
    for_rows(
        g.nr, sc, skip_if_s,
        [&](int q) {
            const Cell e = cell_of(g, 0, q);
            row.load(g, e, q, g.nr, m.U);
            load_matrix<B * B, M>(m.dr + (size_t)q * B * B, dv);
            fine.members(up, e);
        },
        [&](int q) {
            double v[B], x[B];
            fine.load(up);
            red_row<B, ND, M>(row, q, rr, z, v);
            block_mul<B, M>(dv, v, x);
            fine.store(up, x);
        });
}

// z = D_b^-1 (rb - L rr): the sweep from z = 0.
template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_pre_kernel(RbGrid g, RbMatrix<const M> m, const double* rr, const double* rb,
                                                     double* z, const KScal* sc, int skip_if_s)
{
    const int nk = g.n - g.nr;
    StencilRow<B, ND, M> row;
    M dv[B * B];
    for_rows(
        nk, sc, skip_if_s,
        [&](int q) {
            if (rr) row.load(g, cell_of(g, 1, q), q, nk, m.L);
            load_matrix<B * B, M>(m.db + (size_t)q * B * B, dv);
        },
        [&](int q) {
            double acc[B], v[B], x[B];
#pragma unroll
            for (int t = 0; t < B; ++t) acc[t] = 0.0;
            load_bvec<B, double>(rb, q, v);
            if (rr) row.dot(rr, acc);
#pragma unroll
            for (int t = 0; t < B; ++t) v[t] = __dsub_rn(v[t], acc[t]);
            block_mul<B, M>(dv, v, x);
            store_bvec<B, double>(z, q, x);
        });
}

// Coarse right-hand side: the sum of t over the black members of each
// aggregate, g lanes per aggregate in the order of the coarse cells (a
// member's row follows its neighbour's: whole segments), summed by a
// butterfly over the g lanes.  rc: red coarse cells, then black ones.
template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_res_kernel(Aggregates a, RbMatrix<const M> m, const double* rb,
                                                     const double* y, const double* z, double* rc, const KScal* sc,
                                                     int skip_if_s)
{
    const int items = a.coarse.n * a.g, padded = (items + 31) & ~31, lg = a.g == 4 ? 2 : a.g - 1;
    const int nk = a.fine.n - a.fine.nr;
    StencilRow<B, ND, M> row;
    M av[B * B];
    Cell C;
    int c = -1;
    for_rows(
        padded, sc, skip_if_s,
        [&](int it) {
            C = cell_at(a.coarse, it < items ? it >> lg : 0);
            c = it < items ? black_member(a, C.i, C.j, C.k, it & (a.g - 1)) : -1;
            if (c < 0) return;
            row.load(a.fine, cell_at(a.fine, c), c >> 1, nk, m.L);
            load_matrix<B * B, M>(m.abb + (size_t)(c >> 1) * B * B, av);
        },
        [&](int it) {
            double t[B];
#pragma unroll
            for (int v = 0; v < B; ++v) t[v] = 0.0;
            if (c >= 0) {
                double zv[B];
                load_bvec<B, double>(z, c >> 1, zv);
                residual_row<B, ND, M>(row, av, c >> 1, rb, y, zv, t);
            }
            for (int o = 1; o < a.g; o <<= 1)
#pragma unroll
                for (int v = 0; v < B; ++v) t[v] += __shfl_xor_sync(0xffffffffu, t[v], o);
            if (it < items && (it & (a.g - 1)) == 0)
                store_bvec<B, double>(rc, (C.c >> 1) + (((C.i + C.j + C.k) & 1) ? a.coarse.nr : 0), t);
        });
}

// The same of the right-hand side itself (rr null: zero), for a level
// without pre-smoothing: pairs, a black member and the red one beside it.
template <int B>
__global__ void __launch_bounds__(512, 1) rb_restrict_kernel(Aggregates a, const double* rr, const double* rb, double* rc,
                                                          const KScal* sc, int skip_if_s)
{
    for_rows(
        a.coarse.n, sc, skip_if_s, [](int) {},
        [&](int p) {
            const Cell C = cell_at(a.coarse, p);
            double s[B];
#pragma unroll
            for (int t = 0; t < B; ++t) s[t] = 0.0;
            const int i0 = C.i << a.sx, j0 = C.j << a.sy, k0 = C.k << a.sz;
            for (int o = 0; o < (1 << (a.sx + a.sy + a.sz)); ++o) {
                const int i = i0 + (a.sx ? o & 1 : 0), j = j0 + (a.sy ? (o >> a.sx) & 1 : 0),
                          k = k0 + (a.sz ? o >> (a.sx + a.sy) : 0);
                if (i >= a.fine.nx || j >= a.fine.ny || k >= a.fine.nz) continue;
                const double* r = ((i + j + k) & 1) ? rb : rr;
                if (!r) continue;
                double v[B];
                load_bvec<B, double>(r, (i + a.fine.nx * (j + a.fine.ny * k)) >> 1, v);
#pragma unroll
                for (int t = 0; t < B; ++t) s[t] += v[t];
            }
            store_bvec<B, double>(rc, (p >> 1) + (((C.i + C.j + C.k) & 1) ? a.coarse.nr : 0), s);
        });
}

// z += D_b^-1 (rb - A_bb z - L y), handed to the finer level.
template <int B, int ND, class M>
__global__ void __launch_bounds__(512, 1) rb_post_kernel(RbGrid g, RbMatrix<const M> m, const double* rb, const double* y,
                                                      double* z, UpView up, const KScal* sc, int skip_if_s)
{
    const int nk = g.n - g.nr;
    StencilRow<B, ND, M> row;
    UpRow<B> fine;
    M av[B * B], dv[B * B];
    for_rows(
        nk, sc, skip_if_s,
        [&](int q) {
            const Cell e = cell_of(g, 1, q);
            row.load(g, e, q, nk, m.L);
            load_matrix<B * B, M>(m.abb + (size_t)q * B * B, av);
            load_matrix<B * B, M>(m.db + (size_t)q * B * B, dv);
            fine.members(up, e);
        },
        [&](int q) {
            double zv[B], t[B], x[B];
            fine.load(up);
            load_bvec<B, double>(z, q, zv);
            residual_row<B, ND, M>(row, av, q, rb, y, zv, t);
            block_mul<B, M>(dv, t, x);
#pragma unroll
            for (int c = 0; c < B; ++c) zv[c] = __dadd_rn(zv[c], x[c]);
            store_bvec<B, double>(z, q, zv);
            fine.store(up, zv);
        });
}

// The coarsest level: inv r, a warp per unknown (see dense_rows; red cells,
// then black ones), handed to the finer level.
template <int B, class M>
__device__ __forceinline__ void rb_dense_rows(const RbGrid& g, const M* __restrict__ inv, const double* r,
                                              const UpView& up, int tid, int nth)
{
    const int lane = tid & 31, n = g.n * B;
    for (int i = tid >> 5; i < n; i += nth >> 5) {
        double s = 0.0;
        for (int j = lane; j < n; j += 32) s = __fma_rn((double)inv[i * n + j], r[j], s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const int P = i / B, c = i - P * B;
        if (lane < up.agg.g) {
            const Cell e = P < g.nr ? cell_of(g, 0, P) : cell_of(g, 1, P - g.nr);
            const int f = black_member(up.agg, e.i, e.j, e.k, lane);
            if (f >= 0) {
                double* w = up.w + (size_t)(f >> 1) * B + c;
                *w = __fma_rn(up.alpha, s, up.add ? *w : 0.0);
            }
        }
    }
}

template <int B, class M>
__global__ void __launch_bounds__(1024) rb_dense_kernel(RbGrid g, const M* __restrict__ inv, const double* r, UpView up,
                                                        const KScal* sc, int skip_if_s)
{
    pdl_trigger();
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) return;
    rb_dense_rows<B, M>(g, inv, r, up, (int)threadIdx.x, (int)blockDim.x);
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
        StencilRow<B, ND, double> row;
        row.load(g, cell_of(g, 1, q), q, nk, m.L);
        row.dot(b, acc);
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
    rb_spmv_kernel(RbGrid g, RbMatrix<const double> m, const double* z, const double* y, const double* h, double* v,
                   double* partials, unsigned int* counter,
                   KScal* sc)
{
    constexpr int ND_ = OMEGA ? 2 : 1;
    const int nk = g.n - g.nr;
    double d[ND_];
#pragma unroll
    for (int k = 0; k < ND_; ++k) d[k] = 0.0;
    StencilRow<B, ND, double> row;
    double av[B * B];
    const bool ran = for_rows(
        nk, sc, OMEGA,
        [&](int q) {
            row.load(g, cell_of(g, 1, q), q, nk, m.L);
            load_matrix<B * B, double>(m.abb + (size_t)q * B * B, av);
        },
        [&](int q) {
            double acc[B], zv[B], az[B], hv[B];
#pragma unroll
            for (int t = 0; t < B; ++t) acc[t] = 0.0;
            load_bvec<B, double>(z, q, zv);
            load_bvec<B, double>(h, q, hv);
            row.dot(y, acc);
            block_mul<B, double>(av, zv, az);
#pragma unroll
            for (int t = 0; t < B; ++t) acc[t] += az[t];
            store_bvec<B, double>(v, q, acc);
#pragma unroll
            for (int t = 0; t < B; ++t) {
                d[0] += hv[t] * acc[t];
                if (OMEGA) d[ND_ - 1] += acc[t] * acc[t];
            }
        });
    if (!ran) return;  // the same in every block
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
        StencilRow<B, ND, double> row;
        row.load(g, e, q, g.nr, m.U);
        load_matrix<B * B, double>(m.dr + (size_t)q * B * B, dv);
        red_row<B, ND, double>(row, q, b, x, v);
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
// its diagonal entry, at most 1): of the component that is coupled most.  The
// smoothers reduce the others well whatever is paired; with all components
// added up, the weak transport of a two-phase system along x and y halved the
// 25 : 1 of its pressure as soon as there was flow (33x31x17: 14 iterations a
// solve with the pressure's pairs, 18 with those).
template <int B>
__device__ __forceinline__ void strengths(const RbGrid& g, int nd, const double* __restrict__ a, double* partials,
                                          unsigned int* counter, double* out, const SumBlocks& at)
{
    constexpr int bb = B * B;
    const RbMatrix<const double> m(a, nd, bb, g.n, g.nr);
    double sum[3 * B];
#pragma unroll
    for (int t = 0; t < 3 * B; ++t) sum[t] = 0.0;
    for (int P = at.block * kThreads + (int)threadIdx.x; P < g.n; P += at.blocks * kThreads) {
        const bool red = P < g.nr;
        const int rows = red ? g.nr : g.n - g.nr, q = red ? P : P - g.nr;
#pragma unroll
        for (int c = 0; c < B; ++c) {
            const int e = c * B + c;
            const double diag = fabs((red ? m.dr : m.abb)[(size_t)q * bb + e]);
            double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int d = 0; d < 6; ++d)
                if (d < nd) s[d >> 1] += fabs((red ? m.U : m.L)[((size_t)d * rows + q) * bb + e]);
            const double all = s[0] + s[1] + s[2];
            if (!(all > 0.0) || !(diag > 0.0) || !isfinite(all / diag)) continue;
            const double w = fmin(1.0, all / diag) / all;
#pragma unroll
            for (int t = 0; t < 3; ++t) sum[3 * c + t] += w * s[t];
        }
    }
    double s[3 * B];
    if (grid_sum<3 * B>(sum, partials, counter, s, at)) {
        double most = -1.0;
#pragma unroll
        for (int c = 0; c < B; ++c) {
            const double all = s[3 * c] + s[3 * c + 1] + s[3 * c + 2];
            if (!(all > most)) continue;
            most = all;
            for (int t = 0; t < 3; ++t) out[t] = s[3 * c + t];
        }
    }
}

template <int B>
__global__ void __launch_bounds__(kThreads) rb_strength_kernel(RbGrid g, int nd, const double* __restrict__ a,
                                                               double* partials, unsigned int* counter, double* out)
{
    strengths<B>(g, nd, a, partials, counter, out, SumBlocks());
}

// The strengths of the fine matrix by the blocks from `first` on of the launch
// that makes the first coarse one (with a launch of their own a step of heat
// 64x64 took 577 to 583 us, so 575 to 578).
struct StrengthPart {
    int first = 0, blocks = 0;
    double* partials = nullptr;
    unsigned int* counter = nullptr;
    double* out = nullptr;
};

// The coarse matrix R A R^T of a 0/1 aggregation, one thread per value of a
// coarse cell: the blocks of its members that cross each of its faces, and
// its diagonal block with the couplings inside it, summed in the order of
// the members and directions.
template <int B>
__global__ void __launch_bounds__(kThreads) rb_galerkin_kernel(Aggregates a, int nd, const double* __restrict__ fa,
                                                               double* __restrict__ ca, StrengthPart sp)
{
    constexpr int bb = B * B;
    if (sp.blocks && (int)blockIdx.x >= sp.first) {
        strengths<B>(a.fine, nd, fa, sp.partials, sp.counter, sp.out, SumBlocks((int)blockIdx.x - sp.first, sp.blocks));
        return;
    }
    const RbGrid &f = a.fine, &g = a.coarse;
    const RbMatrix<const double> F(fa, nd, bb, f.n, f.nr);
    const RbMatrix<double> G(ca, nd, bb, g.n, g.nr);
    for (int64_t x = (int64_t)blockIdx.x * kThreads + threadIdx.x; x < (int64_t)g.n * bb;
         x += (int64_t)(gridDim.x - sp.blocks) * kThreads) {
        const int c = (int)(x / bb), e = (int)(x - (int64_t)c * bb);
        const Cell C = cell_at(g, c);
        const bool red = ((C.i + C.j + C.k) & 1) == 0;
        const int q = c >> 1, rows = red ? g.nr : g.n - g.nr;
        double diag = 0.0, off[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const int nx = 1 << a.sx, ny = 1 << a.sy, nz = 1 << a.sz;
        for (int dz = 0; dz < nz; ++dz)
            for (int dy = 0; dy < ny; ++dy) {
                // a member and the one beside it, or only it: their loads
                // before the first sum (a missing neighbour's block is zero).
                // A level of a few blocks waits for little else: 13 -> 5.3 us
                double v[2][6], dd[2];
                bool in[2];
#pragma unroll
                for (int dx = 0; dx < 2; ++dx) {
                    Cell m;
                    m.i = (C.i << a.sx) + dx;
                    m.j = (C.j << a.sy) + dy;
                    m.k = (C.k << a.sz) + dz;
                    in[dx] = dx < nx && m.i < f.nx && m.j < f.ny && m.k < f.nz;
                    m.c = in[dx] ? m.i + f.nx * (m.j + f.ny * m.k) : 0;
                    const bool mr = ((m.i + m.j + m.k) & 1) == 0 || !in[dx];
                    const int mq = m.c >> 1, mrows = mr ? f.nr : f.n - f.nr;
                    dd[dx] = (mr ? F.dr : F.abb)[(size_t)mq * bb + e];
#pragma unroll
                    for (int d = 0; d < 6; ++d)
                        v[dx][d] = d < nd ? (mr ? F.U : F.L)[((size_t)d * mrows + mq) * bb + e] : 0.0;
                }
#pragma unroll
                for (int dx = 0; dx < 2; ++dx) {
                    if (!in[dx]) continue;
                    diag += dd[dx];
#pragma unroll
                    for (int d = 0; d < 6; ++d) {
                        // inside the aggregate: the direction is paired and
                        // leads to the other half
                        const bool inner = d < 2 ? a.sx && dx != (d & 1) : d < 4 ? a.sy && dy != (d & 1) : a.sz && dz != (d & 1);
                        if (inner) diag += v[dx][d];
                        else off[d] += v[dx][d];
                    }
                }
            }
        (red ? G.dr : G.abb)[(size_t)q * bb + e] = diag;
#pragma unroll
        for (int d = 0; d < 6; ++d)
            if (d < nd) (red ? G.U : G.L)[((size_t)d * rows + q) * bb + e] = off[d];
    }
}

// The factors need no order between levels, so one launch does all of them:
// blocks [first, first + blocks) take the rows of a level (a launch per level
// and colour was 3.5 to 6.7 us each for the small ones).
struct RbFactorLevel {
    RbGrid g;
    double* a = nullptr;
    int first = 0, blocks = 0;
};

// Every level pairs a direction, so there are at most the sum of ceil(log2
// side) of them below level 0: in 3D less than log2(cells) + 3, and
// two_colour_fits gives cells < 2^31 / 7; in 2D less.
constexpr int kMaxRbLevels = 32;

struct RbFactorParams {
    int nlev = 0;
    RbFactorLevel lv[kMaxRbLevels];
    RbGrid dense;                     // the coarsest level
    const double* dense_a = nullptr;
    double* inverse = nullptr;
    __device__ __forceinline__ const RbFactorLevel& of(int block) const
    {
        int l = 0;
        while (l + 1 < nlev && block >= lv[l + 1].first) ++l;
        return lv[l];
    }
};

// The coarsest matrix, dense and row-major (red cells, then black ones), by
// one block, for dense_inverse_block.
template <int B>
__device__ __forceinline__ void dense_fill(const RbGrid& g, int nd, const double* a, double* dense)
{
    constexpr int BB = B * B;
    const int n = g.n * B, tid = (int)threadIdx.x, nth = (int)blockDim.x;
    const RbMatrix<const double> m(a, nd, BB, g.n, g.nr);
    for (int x = tid; x < n * n; x += nth) dense[x] = 0.0;
    __syncthreads();
    for (int x = tid; x < g.n * (nd + 1); x += nth) {
        const int P = x / (nd + 1), d = x - P * (nd + 1);
        const bool red = P < g.nr;
        const int rows = red ? g.nr : g.n - g.nr, q = red ? P : P - g.nr;
        const Cell e = cell_of(g, red ? 0 : 1, q);
        int nq, Q = P;
        const double* v = (red ? m.dr : m.abb) + (size_t)q * BB;
        if (d < nd) {
            if (!neighbour(g, e, d, nq)) continue;
            Q = red ? g.nr + nq : nq;
            v = (red ? m.U : m.L) + ((size_t)d * rows + q) * BB;
        }
#pragma unroll
        for (int t = 0; t < BB; ++t) dense[(size_t)(P * B + t / B) * n + Q * B + t % B] = v[t];
    }
    __syncthreads();
}

// D_r^-1 over the red cells of all levels.
template <int B>
__global__ void __launch_bounds__(kThreads) rb_factor_red_kernel(const __grid_constant__ RbFactorParams p, int nd,
                                                                int* status)
{
    constexpr int BB = B * B;
    const RbFactorLevel& L = p.of((int)blockIdx.x);
    const RbGrid& g = L.g;
    double* const dr = RbMatrix<double>(L.a, nd, BB, g.n, g.nr).dr;
    for (int64_t q = (int64_t)(blockIdx.x - L.first) * blockDim.x + threadIdx.x; q < g.nr;
         q += (int64_t)L.blocks * blockDim.x) {
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
__global__ void __launch_bounds__(kInverseThreads, 1)
    rb_factor_black_kernel(const __grid_constant__ RbFactorParams p, int* status)
{
    constexpr int BB = B * B;
    if (blockIdx.x == 0) {
        dense_fill<B>(p.dense, ND, p.dense_a, p.inverse);
        dense_inverse_block(p.dense.n * B, p.inverse, status);
        return;
    }
    const RbFactorLevel& L = p.of((int)blockIdx.x);
    const RbGrid& g = L.g;
    const RbMatrix<double> m(L.a, ND, BB, g.n, g.nr);
    const int nk = g.n - g.nr;
    for (int64_t q64 = (int64_t)(blockIdx.x - L.first) * blockDim.x + threadIdx.x; q64 < nk;
         q64 += (int64_t)L.blocks * blockDim.x) {
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

// ---- the coarse end of the cycle in one kernel ----------------------------------
// The levels from one down to the dense solve and back, resident in the shared
// memory of one thread-block cluster: every block holds the matrix rows and
// the vector entries of its share of each level's cells, neighbours' values are
// read from the other blocks' shared memory, and a cluster barrier ends a step.
// A step takes 1.2k to 2.5k cycles, most of it index arithmetic and FP64
// latency (through global memory, two or three round trips to L2 and a barrier
// that waits for the stores to reach it: 2.4k to 9k).  Every step has one call
// site: another copy of its code would be fetched anew, 8k to 10k cycles.  The
// cycle from the 32x32x4 level of two-phase 128x128x64: 33 us through global
// memory, 19 so.  The smallest levels are block 0's alone (solo), with block
// barriers; the dense solve's rows are shared out again.  The matrices are copied in at every launch, before the
// wait for the previous kernel.  Products and sums are those of the one-step
// kernels, in their order; where those add alpha zc to the finer level's z
// (UpRow), the finer level here reads both (z0_at): the same bits.
constexpr int kRbTailSmem = 220 * 1024;
constexpr int kRbSoloCells = 256;  // a level of at most these cells is block 0's

template <class M>
struct RbTailLevel {
    RbGrid g;
    int coarsest = 0, pre = 1;
    int rows = 0;     // rows of a colour that a block holds
    FastDiv by_rows;  // the block of a row
    double alpha = 1.0;
    const M* a = nullptr;  // matrix (RbMatrix), or the dense inverse of the coarsest level
    Aggregates agg;        // to the next level
    int so_m = 0, so_v = 0, vec = 0;  // shared memory: matrix, vectors and a vector's bytes
    int so_r = 0;                     // coarsest level: a copy of its right-hand side
};

template <class M>
struct RbTailParams {
    RbTailLevel<M> lv[kMaxTail];
    int nlev = 0;
    int solo_first = 0;                    // first level that is block 0's (nlev - 1: none)
    const double *rr = nullptr, *rb = nullptr;  // the first level's right-hand side
    double* z = nullptr;                   // where its black rows go when it is level 0
    UpView up;                             // where its rows go otherwise
    long long* trace = nullptr;
};
static_assert(sizeof(RbTailParams<double>) <= 4096, "fused cycle parameters exceed 4 KB");

// A vector over the rows of a colour, spread over the cluster's blocks.
struct RbVec {
    unsigned base;  // shared memory address in every block
    int rows;
    FastDiv by;
};

__device__ __forceinline__ unsigned remote(const RbVec& v, int q, int bytes)
{
    const int owner = v.by(q);
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(v.base + (unsigned)((q - owner * v.rows) * bytes)), "r"(owner));
    return a;
}

template <int B>
__device__ __forceinline__ void load_vec(const RbVec& v, int q, double (&x)[B])
{
    const unsigned a = remote(v, q, 8 * B);
    if constexpr (B == 2) {
        asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(x[0]), "=d"(x[1]) : "r"(a) : "memory");
    } else {
#pragma unroll
        for (int t = 0; t < B; ++t)
            asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x[t]) : "r"(a + 8 * t) : "memory");
    }
}

template <int B>
__device__ __forceinline__ void store_vec(const RbVec& v, int q, const double (&x)[B])
{
    const unsigned a = remote(v, q, 8 * B);
#pragma unroll
    for (int t = 0; t < B; ++t)
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a + 8 * t), "d"(x[t]) : "memory");
}

// A level as a block sees it.
template <int B, int ND, class M>
struct RbTailView {
    static constexpr int BB = B * B;
    const RbTailLevel<M>& L;
    const M *U, *Lo, *dr, *abb, *db;  // this block's rows
    RbVec rr, rb, y, z, t;
    int lo;  // this block's first row of a colour
    __device__ __forceinline__ RbTailView(const RbTailLevel<M>& level, unsigned char* sm, int rank) : L(level)
    {
        U = reinterpret_cast<const M*>(sm + L.so_m);
        Lo = U + (size_t)ND * L.rows * BB;
        dr = Lo + (size_t)ND * L.rows * BB;
        abb = dr + (size_t)L.rows * BB;
        db = abb + (size_t)L.rows * BB;
        const unsigned v = (unsigned)__cvta_generic_to_shared(sm + L.so_v);
        rr = RbVec{v, L.rows, L.by_rows};
        rb = RbVec{v + L.vec, L.rows, L.by_rows};
        y = RbVec{v + 2 * L.vec, L.rows, L.by_rows};
        z = RbVec{v + 3 * L.vec, L.rows, L.by_rows};
        t = RbVec{v + 4 * L.vec, L.rows, L.by_rows};
        lo = rank * L.rows;
    }
    __device__ __forceinline__ int hi(int colour) const
    {
        return min(lo + L.rows, colour ? L.g.n - L.g.nr : L.g.nr);
    }
};

// StencilRow::dot over a block's rows, the neighbours' values from get(neighbour's
// cell, its number, value).
template <int B, int ND, class M, class Get>
__device__ __forceinline__ void tail_dot(const RbGrid& g, const Cell& e, int q, int others, const M* a, int rows, int ql,
                                         Get&& get, double (&acc)[B])
{
    constexpr int BB = B * B;
    M av[ND][BB];
    double xv[ND][B];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        int nq;
        Cell f = e;
        if (neighbour(g, e, d, nq)) {
            const int s = d & 1 ? 1 : -1;
            if (d < 2) f.i += s;
            else if (d < 4) f.j += s;
            else f.k += s;
        } else {
            nq = min(q, others - 1);  // a zero block
        }
        load_block<BB, M>(a + ((size_t)d * rows + ql) * BB, av[d]);
        get(f, nq, xv[d]);
    }
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int i = 0; i < B; ++i)
#pragma unroll
            for (int j = 0; j < B; ++j) acc[i] = __fma_rn((double)av[d][i * B + j], xv[d][j], acc[i]);
}

// z + alpha zc of a black cell (z taken as zero without pre-smoothing): the
// iterate after the coarse correction.
template <int B, int ND, class M>
__device__ __forceinline__ void z0_at(const RbTailView<B, ND, M>& V, const RbTailView<B, ND, M>& C, const Cell& f, int q,
                                      double (&x)[B])
{
    const Aggregates& a = V.L.agg;
    const int ci = f.i >> a.sx, cj = f.j >> a.sy, ck = f.k >> a.sz;
    const int P = ci + a.coarse.nx * (cj + a.coarse.ny * ck);
    double zc[B];
    load_vec<B>(((ci + cj + ck) & 1) ? C.z : C.y, P >> 1, zc);
#pragma unroll
    for (int t = 0; t < B; ++t) x[t] = 0.0;
    if (V.L.pre) load_vec<B>(V.z, q, x);
#pragma unroll
    for (int t = 0; t < B; ++t) x[t] = __fma_rn(V.L.alpha, zc[t], x[t]);
}

// One level's steps down to the coarse right-hand side; sync() ends a step.
template <int B, int ND, class M, class Sync>
__device__ __forceinline__ void tail_down(const RbTailView<B, ND, M>& V, const RbTailView<B, ND, M>& C, bool has_red,
                                          int tid, int nth, Sync&& sync)
{
    constexpr int BB = B * B;
    const RbTailLevel<M>& L = V.L;
    const RbGrid& g = L.g;
    const int nk = g.n - g.nr;
    if (L.pre) {
        for (int q = V.lo + tid; q < V.hi(1); q += nth) {  // rb_pre_kernel
            const int ql = q - V.lo;
            M dv[BB];
            double acc[B], v[B], x[B];
#pragma unroll
            for (int t = 0; t < B; ++t) acc[t] = 0.0;
            load_vec<B>(V.rb, q, v);
            load_block<BB, M>(V.db + (size_t)ql * BB, dv);
            if (has_red)
                tail_dot<B, ND, M>(g, cell_of(g, 1, q), q, g.nr, V.Lo, L.rows, ql,
                                   [&](const Cell&, int nq, double (&w)[B]) { load_vec<B>(V.rr, nq, w); }, acc);
#pragma unroll
            for (int t = 0; t < B; ++t) v[t] = __dsub_rn(v[t], acc[t]);
            block_mul<B, M>(dv, v, x);
            store_vec<B>(V.z, q, x);
        }
        sync();
        for (int q = V.lo + tid; q < V.hi(0); q += nth) {  // rb_y_kernel
            double acc[B], v[B];
#pragma unroll
            for (int t = 0; t < B; ++t) acc[t] = v[t] = 0.0;
            if (has_red) load_vec<B>(V.rr, q, v);
            tail_dot<B, ND, M>(g, cell_of(g, 0, q), q, nk, V.U, L.rows, q - V.lo,
                               [&](const Cell&, int nq, double (&w)[B]) { load_vec<B>(V.z, nq, w); }, acc);
#pragma unroll
            for (int t = 0; t < B; ++t) v[t] = __dsub_rn(v[t], acc[t]);
            store_vec<B>(V.y, q, v);
        }
        sync();
        for (int q = V.lo + tid; q < V.hi(1); q += nth) {  // the residual of rb_res_kernel
            const int ql = q - V.lo;
            M av[BB];
            double acc[B], az[B], z[B], t[B];
#pragma unroll
            for (int c = 0; c < B; ++c) acc[c] = 0.0;
            load_vec<B>(V.rb, q, t);
            load_vec<B>(V.z, q, z);
            load_block<BB, M>(V.abb + (size_t)ql * BB, av);
            tail_dot<B, ND, M>(g, cell_of(g, 1, q), q, g.nr, V.Lo, L.rows, ql,
                               [&](const Cell&, int nq, double (&w)[B]) { load_vec<B>(V.y, nq, w); }, acc);
            block_mul<B, M>(av, z, az);
#pragma unroll
            for (int c = 0; c < B; ++c) t[c] = __dsub_rn(__dsub_rn(t[c], az[c]), acc[c]);
            store_vec<B>(V.t, q, t);
        }
        sync();
    }
    // the coarse rows that this block holds
    const RbGrid& G = C.L.g;
    for (int i = tid; i < 2 * C.L.rows; i += nth) {
        const int colour = i < C.L.rows ? 0 : 1, q = C.lo + i - (colour ? C.L.rows : 0);
        if (q >= C.hi(colour)) continue;
        const Cell e = cell_of(G, colour, q);
        double s[B];
        if (L.pre) {  // the butterfly sum of rb_res_kernel
            double w[4][B];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int c = m < L.agg.g ? black_member(L.agg, e.i, e.j, e.k, m) : -1;
#pragma unroll
                for (int t = 0; t < B; ++t) w[m][t] = 0.0;
                if (c >= 0) load_vec<B>(V.t, c >> 1, w[m]);
            }
#pragma unroll
            for (int t = 0; t < B; ++t)
                s[t] = L.agg.g == 1 ? w[0][t]
                                    : L.agg.g == 2 ? __dadd_rn(w[0][t], w[1][t])
                                                   : __dadd_rn(__dadd_rn(w[0][t], w[1][t]), __dadd_rn(w[2][t], w[3][t]));
        } else {  // rb_restrict_kernel
            const Aggregates& a = L.agg;
#pragma unroll
            for (int t = 0; t < B; ++t) s[t] = 0.0;
            for (int o = 0; o < (1 << (a.sx + a.sy + a.sz)); ++o) {
                const int x = (e.i << a.sx) + (a.sx ? o & 1 : 0), y = (e.j << a.sy) + (a.sy ? (o >> a.sx) & 1 : 0),
                          z = (e.k << a.sz) + (a.sz ? o >> (a.sx + a.sy) : 0);
                if (x >= g.nx || y >= g.ny || z >= g.nz) continue;
                const bool black = (x + y + z) & 1;
                if (!black && !has_red) continue;
                double w[B];
                load_vec<B>(black ? V.rb : V.rr, (x + g.nx * (y + g.ny * z)) >> 1, w);
#pragma unroll
                for (int t = 0; t < B; ++t) s[t] = __dadd_rn(s[t], w[t]);
            }
        }
        store_vec<B>(colour ? C.rb : C.rr, q, s);
    }
    sync();
}

// The steps after the coarse correction: y, the black rows, and the red ones
// unless the level is level 0.  The first level's rows leave the cluster: to
// p.z (level 0) or up the finer level.
template <int B, int ND, class M, class Sync>
__device__ __forceinline__ void tail_up(const RbTailParams<M>& p, const RbTailView<B, ND, M>& V,
                                        const RbTailView<B, ND, M>& C, bool has_red, bool first, int tid, int nth,
                                        Sync&& sync)
{
    const bool need_red = !first || p.z == nullptr;
    const UpView up = first ? p.up : UpView();
    constexpr int BB = B * B;
    const RbTailLevel<M>& L = V.L;
    const RbGrid& g = L.g;
    const int nk = g.n - g.nr;
    for (int q = V.lo + tid; q < V.hi(0); q += nth) {  // rb_y_kernel
        double acc[B], v[B];
#pragma unroll
        for (int t = 0; t < B; ++t) acc[t] = v[t] = 0.0;
        if (has_red) load_vec<B>(V.rr, q, v);
        tail_dot<B, ND, M>(g, cell_of(g, 0, q), q, nk, V.U, L.rows, q - V.lo,
                           [&](const Cell& f, int nq, double (&w)[B]) { z0_at<B, ND, M>(V, C, f, nq, w); }, acc);
#pragma unroll
        for (int t = 0; t < B; ++t) v[t] = __dsub_rn(v[t], acc[t]);
        store_vec<B>(V.y, q, v);
    }
    sync();
    for (int q = V.lo + tid; q < V.hi(1); q += nth) {  // rb_post_kernel
        const int ql = q - V.lo;
        const Cell e = cell_of(g, 1, q);
        M av[BB], dv[BB];
        double acc[B], az[B], z[B], t[B], x[B];
        UpRow<B> fine;
        if (up.w) {
            fine.members(up, e);
            fine.template load<true>(up);
        }
#pragma unroll
        for (int c = 0; c < B; ++c) acc[c] = 0.0;
        z0_at<B, ND, M>(V, C, e, q, z);
        load_vec<B>(V.rb, q, t);
        load_block<BB, M>(V.abb + (size_t)ql * BB, av);
        load_block<BB, M>(V.db + (size_t)ql * BB, dv);
        tail_dot<B, ND, M>(g, e, q, g.nr, V.Lo, L.rows, ql,
                           [&](const Cell&, int nq, double (&w)[B]) { load_vec<B>(V.y, nq, w); }, acc);
        block_mul<B, M>(av, z, az);
#pragma unroll
        for (int c = 0; c < B; ++c) t[c] = __dsub_rn(__dsub_rn(t[c], az[c]), acc[c]);
        block_mul<B, M>(dv, t, x);
#pragma unroll
        for (int c = 0; c < B; ++c) z[c] = __dadd_rn(z[c], x[c]);
        if (need_red) store_vec<B>(V.z, q, z);
        else store_bvec<B, double>(p.z, q, z);
        if (up.w) fine.store(up, z);
    }
    if (!need_red) return;
    sync();
    for (int q = V.lo + tid; q < V.hi(0); q += nth) {  // rb_fin_kernel
        const int ql = q - V.lo;
        const Cell e = cell_of(g, 0, q);
        M dv[BB];
        double acc[B], v[B], x[B];
        UpRow<B> fine;
        if (up.w) {
            fine.members(up, e);
            fine.template load<true>(up);
        }
#pragma unroll
        for (int t = 0; t < B; ++t) acc[t] = v[t] = 0.0;
        load_block<BB, M>(V.dr + (size_t)ql * BB, dv);
        if (has_red) load_vec<B>(V.rr, q, v);
        tail_dot<B, ND, M>(g, e, q, nk, V.U, L.rows, ql,
                           [&](const Cell&, int nq, double (&w)[B]) { load_vec<B>(V.z, nq, w); }, acc);
#pragma unroll
        for (int t = 0; t < B; ++t) v[t] = __dsub_rn(v[t], acc[t]);
        block_mul<B, M>(dv, v, x);
        store_vec<B>(V.y, q, x);  // its right-hand side was read by the rows before the last barrier
        if (up.w) fine.store(up, x);
    }
    sync();
}

// Starts the copy of `bytes` from global to shared memory, both on a boundary
// of PIECE bytes.
template <int PIECE>
__device__ __forceinline__ void copy_in(unsigned dst, const void* src, int bytes, int tid, int nth)
{
    for (int i = tid * PIECE; i < bytes; i += nth * PIECE) {
        if constexpr (PIECE == 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i), "l"((const char*)src + i) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst + i), "l"((const char*)src + i), "n"(PIECE)
                         : "memory");
    }
}

// Starts the copies of this block's rows of every level.
template <int B, int ND, class M>
__device__ __forceinline__ void tail_copies(const RbTailParams<M>& p, unsigned char* sm, int rank, int nblocks)
{
    constexpr int BB = B * B, BLK = BB * (int)sizeof(M);
    constexpr int PIECE = BLK % 16 == 0 ? 16 : BLK % 8 == 0 ? 8 : 4;
    const int tid = (int)threadIdx.x, nth = (int)blockDim.x;
    for (int l = 0; l < p.nlev; ++l) {
        const RbTailLevel<M>& L = p.lv[l];
        unsigned dst = (unsigned)__cvta_generic_to_shared(sm + L.so_m);
        if (L.coarsest) {
            const int n = L.g.n * B, rows = (n + nblocks - 1) / nblocks, r0 = rank * rows;
            if (r0 < n)
                copy_in<(int)sizeof(M)>(dst, L.a + (size_t)r0 * n, min(rows, n - r0) * n * (int)sizeof(M), tid, nth);
            continue;
        }
        const RbMatrix<const M> m(L.a, ND, BB, L.g.n, L.g.nr);
        const int nk = L.g.n - L.g.nr, lo = rank * L.rows;
        const int red = min(L.rows, L.g.nr - lo) * BLK, black = min(L.rows, nk - lo) * BLK;
        const size_t at = (size_t)lo * BB;
        auto part = [&](const M* src, int bytes) {
            if (bytes > 0) copy_in<PIECE>(dst, src, bytes, tid, nth);
            dst += L.rows * BLK;
        };
        for (int d = 0; d < ND; ++d) part(m.U + (size_t)d * L.g.nr * BB + at, red);
        for (int d = 0; d < ND; ++d) part(m.L + (size_t)d * nk * BB + at, black);
        part(m.dr + at, red);
        part(m.abb + at, black);
        part(m.db + at, black);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int B, int ND, class M>
__global__ void __launch_bounds__(kTailThreads, 1)
    rb_tail_kernel(const __grid_constant__ RbTailParams<M> p, const KScal* sc, int skip_if_s)
{
    extern __shared__ __align__(16) unsigned char tail_smem[];
    const int rank = (int)blockIdx.x, nblocks = (int)gridDim.x;  // one cluster
    const int tid = (int)threadIdx.x, nth = (int)blockDim.x;
    // the matrices do not change during a solve: copied before the wait for
    // the previous kernel
    pdl_trigger();
    tail_copies<B, ND, M>(p, tail_smem, rank, nblocks);
    pdl_wait();
    if (mg_skip(sc, skip_if_s)) {  // the same in every block
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    long long* const trace = p.trace;
    int tk = 0;
    if (trace != nullptr && rank == 0 && tid == 0) trace[tk] = clock64();
    ++tk;
    // ends a step: of the cluster, or of block 0 alone (one call site per step,
    // whatever the level: the steps' code is fetched once)
    auto sync_of = [&](bool alone) {
        if (alone) __syncthreads();
        else tail_step(trace, tk);
    };
    auto sync = [&] { tail_step(trace, tk); };
    using View = RbTailView<B, ND, M>;
    auto view = [&](int l) { return View(p.lv[l], tail_smem, rank); };
    const int last = p.nlev - 1, solo = p.solo_first;
    const bool red0 = p.rr != nullptr;
    {
        const View V = view(0);
        double w[B];
        for (int q = V.lo + tid; red0 && q < V.hi(0); q += nth) {
            load_bvec<B, double>(p.rr, q, w);
            store_vec<B>(V.rr, q, w);
        }
        for (int q = V.lo + tid; q < V.hi(1); q += nth) {
            load_bvec<B, double>(p.rb, q, w);
            store_vec<B>(V.rb, q, w);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    sync();
    for (int l = 0; l < last; ++l)
        if (l < solo || rank == 0)
            tail_down<B, ND, M>(view(l), view(l + 1), l > 0 || red0, tid, nth, [&] { sync_of(l >= solo); });
    if (solo < last) sync();
    {  // rb_dense_rows, the right-hand side copied to every block first
        const View V = view(last);
        const int n = V.L.g.n * B, nr = V.L.g.nr, rows = (n + nblocks - 1) / nblocks, lane = tid & 31;
        const M* inv = reinterpret_cast<const M*>(tail_smem + V.L.so_m);
        double* r = reinterpret_cast<double*>(tail_smem + V.L.so_r);
        if (tid < V.L.g.n) {
            double w[B];
            load_vec<B>(tid < nr ? V.rr : V.rb, tid < nr ? tid : tid - nr, w);
            store_bvec<B, double>(r, tid, w);
        }
        __syncthreads();
        for (int k = tid >> 5; k < rows && rank * rows + k < n; k += nth >> 5) {
            double s = 0.0;
            for (int j = lane; j < n; j += 32) s = __fma_rn((double)inv[k * n + j], r[j], s);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) {
                const int i = rank * rows + k, P = i / B, c = i - P * B;
                const unsigned a = remote(P < nr ? V.y : V.z, P < nr ? P : P - nr, 8 * B) + 8 * c;
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(s) : "memory");
            }
        }
        sync();
    }
    for (int l = last - 1; l >= 0; --l) {
        if (l == solo - 1 && solo < last) sync();  // block 0's levels are done
        if (l < solo || rank == 0)
            tail_up<B, ND, M>(p, view(l), view(l + 1), l > 0 || red0, l == 0, tid, nth, [&] { sync_of(l >= solo); });
    }
    cluster_barrier();  // no block leaves while another may read its shared memory
}
