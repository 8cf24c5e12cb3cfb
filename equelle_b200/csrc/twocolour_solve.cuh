// Host side of the two-colour form (twocolour.cuh): hierarchy, set-up, cycle
// and BiCGStab.  Included by solver.cu, inside its anonymous namespace.

#define WITH_ND(nd, ...)            \
    if ((nd) == 4) {                \
        constexpr int ND = 4;       \
        __VA_ARGS__;                \
    } else {                        \
        constexpr int ND = 6;       \
        __VA_ARGS__;                \
    }
#define WITH_RB(an, ...) WITH_BS((an).rb_bs, WITH_ND((an).rb_nd, __VA_ARGS__))

template <class M>
const M* rb_values(const RbLevel& L);
template <>
const double* rb_values<double>(const RbLevel& L) { return (L.coarsest ? L.inv64 : L.a64)->as<double>(); }
template <>
const float* rb_values<float>(const RbLevel& L) { return (L.coarsest ? L.inv32 : L.a32)->as<float>(); }

template <class M>
RbMatrix<const M> rb_matrix(const SolverAnalysis& an, const RbLevel& L)
{
    return RbMatrix<const M>(rb_values<M>(L), an.rb_nd, an.rb_bs * an.rb_bs, L.g.n, L.g.nr);
}

// Levels are coarsened only along the directions at least 1 / kSemiCoarsen
// as strong as the strongest one: the point smoothers do not reduce error
// that varies slowly along a strong direction and quickly along a weak one.
// Krylov ms of two time steps at lines of 4, 6.5, 9 and 13 (before: with
// 2 x 2 x 2 aggregates in the general form), cells of 10 x 10 x dz m:
//   48x48x32    dz 5    13.9  14.1  14.0  14.0  (24.4)
//               dz 3.9  15.6  16.0  15.9  16.0  (27.5)
//               dz 3    15.3  17.2  16.7  20.1  (33.5)
//               dz 2    19.2  16.2  16.3  20.5  (50.7)
//               dz 1    28.8  23.9  23.8  21.4  (101)
//   33x31x17    dz 2    12.9  11.5  11.6  11.6
//   97x83x41    dz 2    37.5  30.9  30.6  38.3
//   256x256  10 x 3.9   10.4  10.0   9.9   9.9  (21.5)
//            10 x 2     23.7  18.2  17.9  20.1  (66.7)
//            10 x 1     43.4  31.8  31.9  30.3  (176)
// 6.5 and 9 choose alike on all of these; 4 pairs one direction too long, 13
// gives up too early.
constexpr double kSemiCoarsen = 6.5;

// The directions that the next level pairs, bit d for direction d, from the
// direction strengths, which are updated to that level's: a coarse cell has
// twice as many fine couplings for every other direction that was paired.
int choose_pairs(const RbGrid& g, double (&strength)[3])
{
    const int dims[3] = {g.nx, g.ny, g.nz};
    double top = 0.0;
    for (int d = 0; d < 3; ++d)
        if (dims[d] > 1) top = std::max(top, strength[d]);
    int s[3], cut = 0;
    for (int d = 0; d < 3; ++d) {
        s[d] = dims[d] > 1 && !(strength[d] * kSemiCoarsen < top) ? 1 : 0;
        cut += s[d];
    }
    for (int d = 0; d < 3; ++d) strength[d] *= std::ldexp(1.0, cut - s[d]);
    return s[0] | s[1] << 1 | s[2] << 2;
}

Aggregates aggregates_of(const RbGrid& g, int pairs)
{
    Aggregates a;
    a.sx = pairs & 1;
    a.sy = pairs >> 1 & 1;
    a.sz = pairs >> 2;
    const int cut = a.sx + a.sy + a.sz;
    a.g = cut > 0 ? 1 << (cut - 1) : 1;
    a.fine = g;
    a.coarse = RbGrid((g.nx + a.sx) >> a.sx, (g.ny + a.sy) >> a.sy, (g.nz + a.sz) >> a.sz);
    return a;
}

// The pairs of every level of a hierarchy whose coarsest level has at most
// `coarsest` unknowns, `bs` per cell.
std::vector<int> choose_hierarchy(RbGrid g, int bs, int coarsest, const double* strength)
{
    double s[3] = {strength[0], strength[1], strength[2]};
    std::vector<int> pairs;
    do {
        pairs.push_back(choose_pairs(g, s));
        g = aggregates_of(g, pairs.back()).coarse;
    } while (g.n * bs > coarsest && g.n > 1);
    return pairs;
}

void rb_gather(Core& c, const SolverAnalysis& an, const double* jval)
{
    const RbLevel& L = an.rb[0];
    const int bb = an.rb_bs * an.rb_bs;
    const int64_t tiles = (L.g.nr + 31) / 32 + (L.g.n - L.g.nr + 31) / 32;
    const double vals = (double)L.g.n * (an.rb_nd + 1) * bb;
    launch(c, "gather_values", [&] {
        rb_gather_kernel<<<(int)std::min<int64_t>(tiles, 148 * 64), kThreads, 0, c.stream>>>(
            L.g, bb, an.rb_nd, an.vmap->as<int>(), jval, L.a64->as<double>());
    }, 12.0 * vals + 8.0 * an.nnz);
}

// The strengths of the gathered matrix's directions (rb_strength_kernel).
void rb_strengths(Core& c, const SolverAnalysis& an)
{
    const RbGrid& g = an.rb[0].g;
    double* out = an.factor_status->as<double>() + 1;
    WITH_BS(an.rb_bs, launch(c, "mg_strength", [&] {
                rb_strength_kernel<BS><<<blocksFor(g.n, kThreads, kRedBlocks), kThreads, 0, c.stream>>>(
                    g, an.rb_nd, an.rb[0].a64->as<double>(), an.partials->as<double>(),
                    an.counter->as<unsigned int>(), out);
            }, 8.0 * an.rb_bs * (an.rb_nd + 1) * g.n));
}

// Waits for what a set-up reports: whether a pivot was zero, and the
// strengths, to c.pinned[1..3] (grids of more than one direction).
bool rb_report(Core& c, const SolverAnalysis& an)
{
    EQG_CUDA(cudaMemcpyAsync(c.pinned, an.factor_status->ptr, 4 * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    int fstat = 0;
    std::memcpy(&fstat, c.pinned, sizeof(int));
    return fstat != 0;
}

// The levels below level 0, as an.rb_pairs says.
void rb_levels(Core& c, SolverAnalysis& an)
{
    const int bs = an.rb_bs, nd = an.rb_nd;
    for (size_t l = 0; l < an.rb_pairs.size(); ++l) {
        RbLevel C;
        {
            RbLevel& F = an.rb[l];
            F.agg = aggregates_of(F.g, an.rb_pairs[l]);
            const int cut = F.agg.sx + F.agg.sy + F.agg.sz;
            F.alpha = c.param_d("linsolver_mg_alpha", cut == 2 && c.nz == 1 ? kMgAlpha2d : kMgAlpha3d);
            // pairs only: no sweep before the correction.  With it, fewer
            // iterations and more time (48x48x32, dz 2: 120 in 16.4 ms against
            // 132 in 16.2; dz 1: 157 in 26.1 against 172 in 23.9; but cells of
            // 2 x 10 x 10: 116 in 15.7 against 136 in 17.1)
            F.pre = cut > 1;
            C.g = F.agg.coarse;
        }
        C.allocate(c, bs, nd);
        if (l + 1 == an.rb_pairs.size()) {
            C.coarsest = true;
            C.inv64 = c.allocN<double>((size_t)C.n * C.n);
        }
        an.rb.push_back(std::move(C));
    }
    if (c.verbose > 2) {
        std::printf("        linear solver: %dx%d blocks, two colours, levels:", bs, bs);
        for (auto& L : an.rb) std::printf(" %dx%dx%d", L.g.nx, L.g.ny, L.g.nz);
        std::printf("\n");
    }
}

// The two-colour hierarchy of a system of `bs` unknowns per cell of the
// Cartesian grid, built on the device; false when its pattern couples cells
// that are no neighbours, or the form has no room for it, or there is no black
// cell (a missing neighbour's value is read from a cell of the other colour).
bool rb_analyse(Core& c, SolverAnalysis& an, const Pattern& p, int bs, int coarsest, const double* jval)
{
    const int nd = c.nz > 1 ? 6 : 4, bb = bs * bs;
    const int64_t cells = (int64_t)c.nx * c.ny * c.nz;
    if (cells < 2 || !two_colour_fits(cells, nd, bb)) return false;
    an.rb_bs = bs;
    an.rb_nd = nd;
    an.rb_coarsest = coarsest;
    an.rb.emplace_back();
    {
        RbLevel& L = an.rb[0];
        L.g = RbGrid(c.nx, c.ny, c.nz);
        const size_t entries = (size_t)L.g.n * (nd + 1) * bb;
        an.vmap = c.allocN<int>(entries);
        Buf bad = c.allocN<int>(1);
        EQG_CUDA(cudaMemsetAsync(an.vmap->ptr, 0xff, entries * sizeof(int), c.stream));
        EQG_CUDA(cudaMemsetAsync(bad->ptr, 0, sizeof(int), c.stream));
        launch(c, "rb_map", [&] {
            rb_map_kernel<<<blocksFor((int64_t)L.g.n * bs), kThreads, 0, c.stream>>>(
                L.g, bs, nd, p.rowptr->as<int>(), p.colind->as<int>(), an.vmap->as<int>(), bad->as<int>());
        });
        int flags = 0;
        EQG_CUDA(cudaMemcpyAsync(c.pinned, bad->ptr, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
        c.sync();
        std::memcpy(&flags, c.pinned, sizeof(int));
        if (flags & 1) {
            an.rb.clear();
            an.vmap = nullptr;
            return false;
        }
        if (bs == 1 && (flags & 2)) {  // a structurally missing diagonal entry
            an.ok = false;
            return true;
        }
    }
    an.partials = c.allocN<double>((size_t)kRedBlocks * 9);
    an.counter = c.allocN<unsigned int>(1);
    EQG_CUDA(cudaMemsetAsync(an.counter->ptr, 0, sizeof(unsigned int), c.stream));
    an.rb[0].allocate(c, bs, nd);
    const RbGrid& g = an.rb[0].g;
    an.rb_directions = (c.nx > 1) + (c.ny > 1) + (c.nz > 1);
    double strength[3] = {1.0, 1.0, 1.0};
    if (an.rb_directions > 1) {
        rb_gather(c, an, jval);
        rb_strengths(c, an);
        rb_report(c, an);
        for (int d = 0; d < 3; ++d) strength[d] = c.pinned[1 + d];
    }
    an.rb_pairs = choose_hierarchy(g, bs, coarsest, strength);
    // the right-hand side, and the BiCGStab vectors of the black half
    an.vec64 = c.allocN<double>(vec_stride(an.n) + 10 * vec_stride((g.n - g.nr) * bs));
    an.multigrid = true;
    rb_levels(c, an);
    return true;
}

// The analysis of the same pattern for other pairs: level 0 and the vectors
// are those of `an`.
std::shared_ptr<SolverAnalysis> rb_repaired(Core& c, const SolverAnalysis& an, std::vector<int> pairs)
{
    auto b = std::make_shared<SolverAnalysis>();
    b->n = an.n;
    b->nnz = an.nnz;
    b->natural = an.natural;
    b->multigrid = true;
    b->rb_bs = an.rb_bs;
    b->rb_nd = an.rb_nd;
    b->rb_coarsest = an.rb_coarsest;
    b->rb_directions = an.rb_directions;
    b->rb_pairs = std::move(pairs);
    b->vmap = an.vmap;
    b->vec64 = an.vec64;
    b->scal = an.scal;
    b->partials = an.partials;
    b->counter = an.counter;
    b->factor_status = an.factor_status;
    b->rb.push_back(an.rb[0]);
    b->rb[0].threads = kThreads;
    rb_levels(c, *b);
    return b;
}

// Matrices of every level and their factors from the Jacobian's values.
void rb_setup(Core& c, SolverAnalysis& an, const double* jval, bool mixed)
{
    const int bs = an.rb_bs, bb = bs * bs, nd = an.rb_nd;
    int* status = an.factor_status->as<int>();
    rb_gather(c, an, jval);
    for (size_t l = 0; l + 1 < an.rb.size(); ++l) {
        const RbLevel &F = an.rb[l], &C = an.rb[l + 1];
        StrengthPart sp;
        sp.first = blocksFor((int64_t)C.g.n * bb);
        if (l == 0 && an.rb_directions > 1) {
            sp.blocks = blocksFor(F.g.n, kThreads, kRedBlocks);
            sp.partials = an.partials->as<double>();
            sp.counter = an.counter->as<unsigned int>();
            sp.out = an.factor_status->as<double>() + 1;
        }
        WITH_BS(bs, launch(c, "mg_galerkin", [&] {
                    rb_galerkin_kernel<BS><<<sp.first + sp.blocks, kThreads, 0, c.stream>>>(
                        F.agg, nd, F.a64->as<double>(), C.a64->as<double>(), sp);
                }, 8.0 * bb * (nd + 1) * ((double)F.g.n + C.g.n)));
    }
    // the levels' factors, and beside them the coarsest one's inverse: one
    // block's chain of n steps (183 us for n = 128, 67 us for n = 60) that the
    // black rows of the other levels run beside, where it waited for two
    // launches a level.  Set-up of a step's solves, before and so: two-phase
    // 48x40 0.66 -> 0.39 ms, 512x512 1.52 -> 1.07, 128x128x64 3.36 -> 2.17
    RbFactorParams red, black;
    double red_bytes = 0.0, black_bytes = 0.0;
    int red_blocks = 0, black_blocks = 1;
    if (an.rb.size() > (size_t)kMaxRbLevels) fail(EQG_ERR_UNSUPPORTED, "linear system with too many levels");
    for (const RbLevel& L : an.rb) {
        if (L.coarsest) {
            black.dense = L.g;
            black.dense_a = L.a64->as<double>();
            black.inverse = L.inv64->as<double>();
            black_bytes += 16.0 * L.n * L.n;
            continue;
        }
        const int nr = L.g.nr, nk = L.g.n - nr;
        RbFactorLevel f;
        f.g = L.g;
        f.a = L.a64->as<double>();
        f.first = red_blocks;
        f.blocks = blocksFor(nr);
        red_blocks += f.blocks;
        red.lv[red.nlev++] = f;
        f.first = black_blocks;
        f.blocks = blocksFor(nk, kInverseThreads);
        black_blocks += f.blocks;
        black.lv[black.nlev++] = f;
        red_bytes += 16.0 * bb * nr;
        black_bytes += 8.0 * bb * (nk * (2.0 * nd + 2.0) + nr * (nd + 1.0));
    }
    if (red.nlev)
        WITH_BS(bs, launch(c, "rb_factor_red", [&] {
                    rb_factor_red_kernel<BS><<<red_blocks, kThreads, 0, c.stream>>>(red, nd, status);
                }, red_bytes));
    WITH_RB(an, launch(c, "rb_factor_black", [&] {
                rb_factor_black_kernel<BS, ND><<<black_blocks, kInverseThreads, 0, c.stream>>>(black, status);
            }, black_bytes));
    if (!mixed) return;
    for (auto& L : an.rb) {
        if (L.coarsest) to_float(c, L.inv64, L.inv32, (int64_t)L.n * L.n);
        else to_float(c, L.a64, L.a32, L.vals);
    }
}

// ---- the cycle -------------------------------------------------------------------
// The vectors of one level.  Level 0 works on the caller's black vectors, its
// red right-hand side is zero.
struct RbVectors {
    const double *rr, *rb;
    double *z, *y;
    UpView up;
    RbVectors(const SolverAnalysis& an, size_t l, const double* in, double* out)
    {
        const RbLevel& L = an.rb[l];
        const size_t red = (size_t)L.g.nr * an.rb_bs;
        double* v = L.v64->as<double>();
        rr = l == 0 ? nullptr : v;
        rb = l == 0 ? in : v + red;
        y = v + L.n;
        z = l == 0 ? out : y + red;
        if (l > 0) {
            const RbLevel& F = an.rb[l - 1];
            up.agg = F.agg;
            up.add = F.pre ? 1 : 0;
            up.alpha = F.alpha;
            up.w = l == 1 ? out : F.v64->as<double>() + F.n + (size_t)F.g.nr * an.rb_bs;
        }
    }
};

// The levels that a cluster of `cl` blocks holds in shared memory: from the
// coarsest one upward, of at most linsolver_mg_fuse_rows unknowns (0: none),
// while every block's share fits in kRbTailSmem bytes.  Returns the first one
// (-1: none) and the bytes of a block; fills the layout.  The levels of at
// most kRbSoloCells cells are block 0's (linsolver_mg_local=0: none).
template <class M>
int plan_rb_tail(Core& c, const SolverAnalysis& an, int cl, int& bytes, RbTailParams<M>* p)
{
    const int nl = (int)an.rb.size(), fuse_rows = c.param_i("linsolver_mg_fuse_rows", 40000);
    const int solo_cells = c.param_i("linsolver_mg_local", 1) ? kRbSoloCells : 0, bs = an.rb_bs;
    auto al = [](int64_t b) { return (b + 15) & ~(int64_t)15; };
    int64_t off = 0;
    int first = -1;
    RbTailParams<M> q;
    int solo = nl - 1;
    for (int l = nl - 1; l >= 0 && nl - l <= kMaxTail; --l) {
        const RbLevel& L = an.rb[l];
        if (!L.coarsest && L.n > fuse_rows) break;
        const bool alone = !L.coarsest && L.g.n <= solo_cells;
        // the coarsest level's vectors are where the level above restricts to
        const bool vectors_alone = alone || (L.coarsest && l > 0 && an.rb[l - 1].g.n <= solo_cells);
        RbTailLevel<M>& t = q.lv[l - std::max(0, nl - kMaxTail)];
        t.g = L.g;
        t.coarsest = L.coarsest ? 1 : 0;
        t.pre = L.pre ? 1 : 0;
        t.alpha = L.alpha;
        t.a = rb_values<M>(L);
        t.agg = L.agg;
        t.rows = vectors_alone ? L.g.nr : (L.g.nr + cl - 1) / cl;
        t.by_rows = FastDiv((unsigned)t.rows);
        t.vec = (int)al((int64_t)t.rows * bs * sizeof(double));
        const int64_t mat = L.coarsest ? (int64_t)((L.n + cl - 1) / cl) * L.n
                                       : (int64_t)(2 * an.rb_nd + 3) * t.rows * bs * bs;
        const int64_t need = al(mat * (int64_t)sizeof(M)) + 5 * (int64_t)t.vec +
                             (L.coarsest ? al((int64_t)L.n * sizeof(double)) : 0);
        // levels of more rows are spread over the whole GPU, one launch per
        // step.  Microseconds an iteration with lines of 128, 256, 512 and 4096
        // rows: two-phase 97x83x41 mixed 215, 215, 224, 223; 512x512 mixed 173,
        // 171, 174, 175; 255x257 mixed 132, 128, 128, 138; 128x128 mixed 91, 91,
        // 83, 83; heat 1000x701 217, 217, 212, 214; 400x300 131, 124, 122, 124
        if (!alone && !L.coarsest && t.rows > kTailThreads / 2 && cl > 1) break;
        if (off + need > kRbTailSmem) break;
        t.so_m = (int)off;
        t.so_v = (int)(off + al(mat * (int64_t)sizeof(M)));
        t.so_r = t.so_v + 5 * t.vec;
        off += need;
        if (alone) solo = l;
        if (!L.coarsest) first = l;
    }
    if (first < 0) return -1;
    bytes = (int)off;
    if (p) {
        p->nlev = nl - first;
        p->solo_first = solo - first;
        for (int i = 0; i < p->nlev; ++i) p->lv[i] = q.lv[first + i - std::max(0, nl - kMaxTail)];
    }
    return first;
}

template <class M>
void launch_rb_tail(Core& c, const SolverAnalysis& an, const double* in, double* out, const KScal* sc, int skip)
{
    const int cl = an.tail_cluster[pc_mode<double, M>()];
    RbTailParams<M> p;
    int smem = 0;
    if (plan_rb_tail<M>(c, an, cl, smem, &p) != an.tail_first) fail(EQG_ERR_DEVICE, "fused coarse cycle: another plan");
    const RbVectors v(an, an.tail_first, in, out);
    p.rr = v.rr;
    p.rb = v.rb;
    p.up = v.up;
    if (an.tail_first == 0) p.z = v.z;
    double bytes = 0.0;
    for (size_t l = an.tail_first; l < an.rb.size(); ++l) {
        const RbLevel& L = an.rb[l];
        bytes += (double)(L.coarsest ? (int64_t)L.n * L.n : L.vals) * sizeof(M) + 4.0 * L.n * sizeof(double);
    }
    if (an.tail_trace) p.trace = an.tail_trace->as<long long>();
    TailLaunch cfg(c, cl, smem);
    WITH_RB(an, launch(c, "rb_tail", [&] {
                EQG_CUDA(cudaLaunchKernelEx(&cfg.cfg, rb_tail_kernel<BS, ND, M>, p, sc, skip));
            }, bytes));
}

// out = V-cycle(in) on the black rows, from level l down.
template <class M>
void rb_cycle(Core& c, const SolverAnalysis& an, size_t l, const double* in, double* out, const KScal* sc, int skip)
{
    if ((int)l == an.tail_first) {
        launch_rb_tail<M>(c, an, in, out, sc, skip);
        return;
    }
    const RbLevel& L = an.rb[l];
    const RbVectors v(an, l, in, out);
    if (L.coarsest) {
        WITH_BS(an.rb_bs, launch(c, "rb_dense", [&] {
                    launch_k(c, rb_dense_kernel<BS, M>, 1, 1024, L.g, rb_values<M>(L), v.rr, v.up, sc, skip);
                }, (double)L.n * L.n * sizeof(M) + 2.0 * L.n * sizeof(double)));
        return;
    }
    double* rc = an.rb[l + 1].v64->as<double>();
    const RbMatrix<const M> m = rb_matrix<M>(an, L);
    const int nr = L.g.nr, nk = L.g.n - nr, nt = L.threads;
    // algorithmic bytes: the stored blocks of a half, the diagonal blocks, and
    // every vector element read or written once
    const double row = 8.0 * an.rb_bs, blk = (double)sizeof(M) * an.rb_bs * an.rb_bs, coarse = row * L.agg.coarse.n;
    const double half_u = an.rb_nd * blk * nr, half_l = an.rb_nd * blk * nk, red = l == 0 ? 0.0 : row * nr;
    auto y_rows = [&] {
        WITH_RB(an, launch(c, "rb_y", [&] {
                    launch_k(c, rb_y_kernel<BS, ND, M>, blocksFor(nr, nt), nt, L.g, m, v.rr, (const double*)v.z, v.y, sc,
                             skip);
                }, half_u + red + row * (nr + nk)));
    };
    if (L.pre) {
        WITH_RB(an, launch(c, "rb_pre", [&] {
                    launch_k(c, rb_pre_kernel<BS, ND, M>, blocksFor(nk, nt), nt, L.g, m, v.rr, v.rb, v.z, sc, skip);
                }, (l == 0 ? 0.0 : half_l) + red + (blk + 2 * row) * nk));
        y_rows();
        WITH_RB(an, launch(c, "rb_res", [&] {
                    launch_k(c, rb_res_kernel<BS, ND, M>, blocksFor((int64_t)L.agg.coarse.n * L.agg.g, nt), nt, L.agg, m,
                             v.rb, (const double*)v.y, (const double*)v.z, rc, sc, skip);
                }, half_l + (blk + 2 * row) * nk + row * nr + coarse));
    } else {
        WITH_BS(an.rb_bs, launch(c, "rb_restrict", [&] {
                    launch_k(c, rb_restrict_kernel<BS>, blocksFor(L.agg.coarse.n, nt), nt, L.agg, v.rr, v.rb, rc, sc,
                             skip);
                }, row * nk + red + coarse));
    }
    rb_cycle<M>(c, an, l + 1, in, out, sc, skip);
    y_rows();
    const double to_fine = v.up.w ? row * v.up.agg.g * (v.up.add ? 2.0 : 1.0) : 0.0;
    WITH_RB(an, launch(c, "rb_post", [&] {
                launch_k(c, rb_post_kernel<BS, ND, M>, blocksFor(nk, nt), nt, L.g, m, v.rb, (const double*)v.y, v.z, v.up,
                         sc, skip);
            }, half_l + (2 * blk + 3 * row + to_fine) * nk + row * nr));
    if (v.up.w == nullptr) return;
    WITH_RB(an, launch(c, "rb_fin", [&] {
                launch_k(c, rb_fin_kernel<BS, ND, M>, blocksFor(nr, nt), nt, L.g, m, v.rr, (const double*)v.z, v.up, sc,
                         skip);
            }, half_u + (blk + row + to_fine) * nr + row * nk));
}

// Chooses the cluster size and the levels of the fused cycle; called before
// any capture.
template <class M>
void prepare_rb_tail(Core& c, SolverAnalysis& an)
{
    const int mode = pc_mode<double, M>();
    int& cl = an.tail_cluster[mode];
    if (!cl) WITH_RB(an, cl = tail_cluster_size(c, rb_tail_kernel<BS, ND, M>, kRbTailSmem));
    int bytes = 0;
    an.tail_first = plan_rb_tail<M>(c, an, cl, bytes, nullptr);
    an.last_mode = mode;
}

// BiCGStab on the black half, M the type of the preconditioner's matrices:
// the solution of A x = rhs, both in the natural order.
template <class M>
SolveResult bicgstab_rb(Core& c, SolverAnalysis& an, const double* rhs, double* xout, double tol, int max_iter,
                        int check_every)
{
    const RbLevel& L0 = an.rb[0];
    const RbGrid& g = L0.g;
    const int bs = an.rb_bs, nr = g.nr, nk = g.n - nr, n = nk * bs;
    double* b = an.vec64->as<double>();
    const Vecs<double> v = vecs<double>(b + vec_stride(an.n), n);
    KScal* sc = an.scal->as<KScal>();
    double* part = an.partials->as<double>();
    unsigned int* cnt = an.counter->as<unsigned int>();
    const RbMatrix<const double> m = rb_matrix<double>(an, L0);
    double* y = L0.v64->as<double>() + L0.n;
    const int nbv = blocksFor(n, kThreads, kRedBlocks), nbk = blocksFor(nk, kThreads, kRedBlocks);
    const double vb = 8.0 * n, yb = 8.0 * nr * bs, blk = 8.0 * bs * bs;
    const double half_u = an.rb_nd * blk * nr, half_l = an.rb_nd * blk * nk;
    WITH_BS(bs, launch(c, "permute", [&] {
                rb_permute_kernel<BS><<<blocksFor(g.n), kThreads, 0, c.stream>>>(g, rhs, b);
            }, 16.0 * an.n));
    WITH_RB(an, launch(c, "rb_init", [&] {
                rb_init_kernel<BS, ND><<<blocksFor(nr, kThreads, kRedBlocks), kThreads, 0, c.stream>>>(
                    g, m, b, v.r, v.rhat, v.p, v.v, v.x, part, cnt, sc, tol * tol);
            }, half_l + vb * 6.0 + yb));
    auto product = [&](const double* z, const double* h, double* out, bool omega) {
        WITH_RB(an, launch(c, "rb_spmv_y", [&] {
                    launch_k(c, rb_y_kernel<BS, ND, double>, blocksFor(nr, L0.threads), L0.threads, g, m,
                             (const double*)nullptr, z, y, (const KScal*)sc, (int)omega);
                }, half_u + vb + yb));
        WITH_RB(an, launch(c, omega ? "rb_spmv_omega" : "rb_spmv_alpha", [&] {
                    launch_k(c, omega ? rb_spmv_kernel<BS, ND, true> : rb_spmv_kernel<BS, ND, false>, nbk, kThreads, g, m,
                             z, (const double*)y, h, out, part, cnt, sc);
                }, half_l + blk * nk + yb + 3.0 * vb));
    };
    auto iteration = [&] {
        launch(c, "bicg_p", [&] {
            launch_k(c, bicg_p_kernel<double>, blocksFor(n), kThreads, (const double*)v.r, (const double*)v.v, v.p, n,
                     (const KScal*)sc);
        }, 4.0 * vb);
        rb_cycle<M>(c, an, 0, v.p, v.ph, sc, 0);
        product(v.ph, v.rhat, v.v, false);
        launch(c, "bicg_s", [&] {
            launch_k(c, bicg_s_kernel<double>, nbv, kThreads, (const double*)v.r, (const double*)v.v, v.s, n, part, cnt,
                     sc);
        }, 3.0 * vb);
        rb_cycle<M>(c, an, 0, v.s, v.sh, sc, 1);
        product(v.sh, v.s, v.t, true);
        launch(c, "bicg_xr", [&] {
            launch_k(c, bicg_xr_kernel<double>, nbv, kThreads, (const double*)v.ph, (const double*)v.sh,
                     (const double*)v.s, (const double*)v.t, (const double*)v.rhat, v.x, v.r, n, part, cnt, sc);
        }, 8.0 * vb);
    };
    autotune<double, M>(c, an, [&] { rb_cycle<M>(c, an, 0, v.r, v.ph, sc, 0); });
    const SolveResult res =
        run_iterations(c, an, sizeof(M) == sizeof(double) ? 0 : 2, tol, max_iter, check_every, iteration);
    WITH_RB(an, launch(c, "rb_solution", [&] {
                rb_solution_kernel<BS, ND><<<blocksFor(nr), kThreads, 0, c.stream>>>(g, m, b, v.x, xout);
            }, half_u + blk * nr + 3.0 * vb + 2.0 * yb));
    return res;
}
