// pm_pair_rows.cuh -- K9 / K10: the FP64 pair kernels, row by row (included
// after pm_pair_col.cuh).  What a row adds up (forces, molecular
// virial, the backward pass) is an operation of its own (ForceRow, MolvirRow,
// AdjRow), run over the column list (K9' / K10', boxes of at least twice the
// cutoff) or over the cell-sorted clusters (K9 / K10, smaller boxes: below).
//
// Over the columns (col_rows64): the list, the test phase and the rings of
// pm_pair_col.cuh; a warp takes rows, or shares of their entries, in a fixed
// order, so that the FP64 energy records do not depend on where the list
// kernel placed a row's entries.  A row whose entries did not fit the list
// gathers them again here, a block at a time: the FP64 forces need no
// capacity, and their sums do not depend on it.
//
// A row is one 8-atom cluster of the cell-sorted order.  A warp takes a row
// (or one of `rows_split` shares of its neighbour cells), and visits every
// atom j of the cell itself and of all its neighbour-cell deltas: every
// ordered pair of the reference's cell pairs once, so each row atom gathers
// its own sums in registers and no other atom's are written.  Two phases
// alternate:
//
//   test   32 candidates per step (lane l: row atom l % 8, candidate l / 8 of
//          a 4-atom half cluster), the minimal-image distance from 32-bit
//          fixed-point coordinates in FP32.  Clusters whose bounding box is
//          beyond the cutoff are left out before (not in the small-grid mode,
//          where a cell pair has no single image).  A distance within the
//          guard band of the cutoff is decided in FP64 in the reference's
//          operation order, so the pair set is the reference's.  Pairs inside
//          go to the row atom's ring in shared memory.
//   pairs  the four lanes of a row atom take the next four of its ring: the
//          FP64 terms run on full warps.
//
// What bounds it: the FP64 pipe in the pair phase (about 120 FP64
// instructions per ordered pair, two issue cycles each), the FP32 test phase
// beside it.  Why rows and rings: over 32 x 32 blocks of two cells only one
// lane in seven held a pair inside the cutoff while the warp ran its ~250
// FP64 instructions (cells half a cutoff wide are filled to two thirds, and a
// third of a cell pair's pairs are inside); visiting each pair from both
// sides doubles the useful pairs and drops the other atom's shared-memory
// sums, and the rings keep every lane of the pair phase busy.
// Measured on the 14,281-atom box: 595 us over cell blocks, 479 us over these
// rows (270 us of it the test phase: partly filled clusters of half-cutoff
// cells, gathered in the kernel).  The column rows take 169 us: prebuilt
// entries of full clusters (half the test), and every pair once, the j side
// added in 64-bit integers by the lane that has it (278 us with every pair from
// both sides, 191 us at four blocks per SM instead of five).  192,003 atoms with
// look-up tables: 5.32 -> 1.27 ms.

constexpr int kRing = 64;            // ring places per row atom
constexpr int kRingDrain = 32;       // a drain stops when every ring is below this

// the largest number of shares a row is cut into (small systems)
constexpr int kRowsSplitMax = 16;

struct RowsShared {
    int ring[kRing * kCluster];      // [place][row atom]: a quarter warp reads eight different banks
    int pre[33];
    int4 cand[32];                   // per lane: first cluster, first slot, end slot, cell offset index
};

struct RowTile { int4 a, b; };       // a lane's two candidates of a cluster

// the row loop: op.begin(slot, valid), op.pair(valid, slot | modified << 30),
// op.end(slot, valid) for every share of a row.  DIFFMOL: pairs of different
// molecules only.
template <bool DIFFMOL, class Op>
__device__ __forceinline__ void cell_rows(const PairArgs& p, RowsShared& sh, Op& op)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, il = lane & 7, jj = lane >> 3;
    const unsigned below = (1u << (8 * jj)) - 1u;
    const CellGrid& cg = p.grid;
    const int split = p.rows_split;
    const int nk = p.nd + 1;
    const int n_items = p.cstart[cg.ncell] * split;
    const float sx = p.lx * 2.3283064365386963e-10f, sy = p.ly * 2.3283064365386963e-10f,
                sz = p.lz * 2.3283064365386963e-10f;          // L / 2^32
    const float far2 = p.cut2f * (1.0f + p.guard), band2 = p.cut2f * (1.0f - p.guard);
    const float lim = p.cut2f * (1.0f + 8.0f * p.guard) + 1e-3f;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < n_items; item += warps) {
        const int row = item / split, part = item - row * split;
        const int A = p.ccell[row];
        const int s0 = p.start[A] + kCluster * (row - p.cstart[A]);
        const int ni = min(kCluster, p.start[A + 1] - s0);
        const bool vi = il < ni;
        const int si = s0 + min(il, ni - 1);
        const int4 Pi = p.sfix[si];
        const float4 ilo = p.cbox[2 * row], ihi = p.cbox[2 * row + 1];
        const int ax = A / (cg.ny * cg.nz), ay = (A / cg.nz) % cg.ny, az = A % cg.nz;
        const int kb = (int)((long long)nk * part / split), ke = (int)((long long)nk * (part + 1) / split);
        op.begin(si, vi);
        int head = 0, cnt = 0;                        // the row atom's ring (the same in its four lanes)

        auto take = [&](const int4& Pj, int j, bool valid) {
            const float dx = (float)(int)((unsigned)Pj.x - (unsigned)Pi.x) * sx;
            const float dy = (float)(int)((unsigned)Pj.y - (unsigned)Pi.y) * sy;
            const float dz = (float)(int)((unsigned)Pj.z - (unsigned)Pi.z) * sz;
            const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
            const bool same = Pj.w == Pi.w;
            bool in = valid && j != si && r2 <= far2 && !(DIFFMOL && same);
            int code = j;
            const bool rare = in && (r2 >= band2 || (!DIFFMOL && same));
            if (__any_sync(FULL, rare)) {
                if (rare) {
                    const int oi = p.smeta[si].x, oj = p.smeta[j].x;
                    if (r2 >= band2) in = !(exact_d2(p, min(oi, oj), max(oi, oj)) > p.cut2d);
                    if (!DIFFMOL && same) {
                        const int x = excl_class(p, oi, oj);
                        if (x == PMGPU_EXCL_FULL) in = false;
                        if (x == PMGPU_EXCL_MODIFIED) code |= 1 << 30;
                    }
                }
            }
            const unsigned b = (__ballot_sync(FULL, in) >> il) & 0x01010101u;
            if (in) sh.ring[((head + cnt + __popc(b & below)) & (kRing - 1)) * kCluster + il] = code;
            cnt += __popc(b);
        };
        auto run = [&]() {                            // the next (up to) four of every ring
            const bool valid = jj < cnt;
            const int e = valid ? sh.ring[((head + jj) & (kRing - 1)) * kCluster + il] : 0;
            op.pair(valid, e);
            const int n = min(4, cnt);
            head = (head + n) & (kRing - 1);
            cnt -= n;
        };

        for (int k0 = kb; k0 < ke; k0 += 32) {
            // one neighbour cell per lane (k = 0: the cell itself)
            const int k = k0 + lane;
            int nc = 0;
            int4 cd = make_int4(0, 0, 0, 0);
            if (k < ke) {
                int B = A;
                if (k > 0) {
                    const int4 d = p.deltas[k - 1];
                    int bx = ax + d.x, by = ay + d.y, bz = az + d.z;
                    bx = ((bx % cg.nx) + cg.nx) % cg.nx;
                    by = ((by % cg.ny) + cg.ny) % cg.ny;
                    bz = ((bz % cg.nz) + cg.nz) % cg.nz;
                    B = (bx * cg.ny + by) * cg.nz + bz;
                }
                const int c0 = p.cstart[B];
                nc = p.cstart[B + 1] - c0;
                cd = make_int4(c0, p.start[B], p.start[B + 1], k);
            }
            int incl = nc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += v;
            }
            __syncwarp();
            sh.cand[lane] = cd;
            sh.pre[lane + 1] = incl;
            if (lane == 0) sh.pre[0] = 0;
            __syncwarp();
            const int total = __shfl_sync(FULL, incl, 31);
            const bool last_round = k0 + 32 >= ke;
            for (int f0 = 0; f0 == 0 || f0 < total; f0 += 32) {
                // the cells' clusters, one per lane: its box against the row's
                const int f = f0 + lane;
                bool near = false;
                int jfirst = 0, nj = 0;
                if (f < total) {
                    int lo = 0, hi = 32;
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (sh.pre[mid] <= f) lo = mid; else hi = mid;
                    }
                    const int4 c = sh.cand[lo];
                    const int u = f - sh.pre[lo];
                    jfirst = c.y + kCluster * u;
                    nj = min(kCluster, c.z - jfirst);
                    near = true;
                    if (!p.wrap) {
                        const float4 o = c.w > 0 ? p.doff[c.w - 1] : make_float4(0.f, 0.f, 0.f, 0.f);
                        near = box_near(ilo, ihi, p.cbox[2 * (c.x + u)], p.cbox[2 * (c.x + u) + 1], o.x, o.y, o.z, lim);
                    }
                }
                unsigned m = __ballot_sync(FULL, near);
                int code = jfirst | (nj << 27);       // nj <= 8, slots below 2^27
                RowTile nt = {make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)};
                auto load = [&](unsigned left, RowTile& t) {
                    const int c = __shfl_sync(FULL, code, left ? __ffs(left) - 1 : 0);
                    const int j0 = c & 0x7ffffff, n = (int)((unsigned)c >> 27);
                    if (left) {
                        t.a = __ldg(p.sfix + j0 + min(jj, n - 1));
                        t.b = __ldg(p.sfix + j0 + min(jj + 4, n - 1));
                    }
                };
                load(m, nt);
                while (true) {
                    // (one copy of the pair phase: the code is large)
                    const bool end = !m && last_round && f0 + 32 >= total;
                    if (end || __any_sync(FULL, cnt > kRing - 8)) {
                        __syncwarp();
                        const int keep = end ? 1 : kRingDrain;
                        while (__any_sync(FULL, cnt >= keep)) run();
                        __syncwarp();
                    }
                    if (!m) break;
                    const RowTile t = nt;
                    const int c = __shfl_sync(FULL, code, __ffs(m) - 1);
                    const int j0 = c & 0x7ffffff, n = (int)((unsigned)c >> 27);
                    m &= m - 1;
                    load(m, nt);                      // the next cluster's, while this one is tested
                    take(t.a, j0 + jj, vi && jj < n);
                    if (n > 4) take(t.b, j0 + jj + 4, vi && jj + 4 < n);
                }
            }
        }
        op.end(si, vi);
        __syncwarp();
    }
}

// slot data of the two layouts: raw position and charge; original index,
// type, molecule
template <bool COL>
__device__ __forceinline__ double4 row_pos(const PairArgs& p, int slot) { return COL ? p.c64[slot] : p.spos64[slot]; }
template <bool COL>
__device__ __forceinline__ int4 row_meta(const PairArgs& p, int slot)
{
    if (!COL) return p.smeta[slot];
    const int4 m = p.cm[slot];
    return make_int4(m.w, m.z, p.cq[slot].w, 0);
}
template <bool COL>
__device__ __forceinline__ int row_type(const PairArgs& p, int slot) { return COL ? p.cm[slot].z : p.smeta[slot].y; }

// d of the pair's nearest image in FP64: the raw difference less the nearest
// whole number of box edges (an edge times -1, 0 or 1 is exact, so this is
// minimalDifference's value bit for bit for atoms within one box edge)
__device__ __forceinline__ double image_diff(double a, double b, double edge, double inv)
{
    const double d = __dadd_rn(b, -a);
    const double big = 6755399441055744.0;           // 1.5 2^52: rounds to an integer
    const double t = __dadd_rn(__fma_rn(d, inv, big), -big);
    return __fma_rn(-t, edge, d);
}

// ---------------------------------------------------------------- rows over the columns
struct ColRowsShared {
    int ring[kColRing * kCluster];
    int ent[kColBlock + 4];
};

// a row operation behind the interface of col_entries: one pair per lane and
// step, four of every ring
template <class RowOp>
struct ColOp64 {
    static constexpr int kKeep = 16;
    static constexpr bool kLocal = false;
    RowOp& op;

    __device__ __forceinline__ void begin(const ColRow& r) { op.begin(r.si, r.vi); }
    __device__ __forceinline__ void drain(ColRow& r, const int* ring, int keep)
    {
        // (the order of ColForce32::drain, in fours)
        const int lane = threadIdx.x & 31, il = lane & 7, jj = lane >> 3;
        const int cnt = r.tail - r.head;
        int m = keep ? cnt >> 2 : (cnt + 3) >> 2;
        int steps = __reduce_max_sync(0xffffffffu, m);
        if (keep) steps = max(1, steps - 4);
        m = min(m, steps);
        int b = m > 0 ? (2 * il) % m : 0;
        bool valid = false;
        auto code = [&](int s) {
            const int at = 4 * b + jj;
            valid = s < m && at < cnt;
            b = b + 1 < m ? b + 1 : 0;
            return valid ? ring[((r.head + at) & (kColRing - 1)) * kCluster + il] : r.si;
        };
        if constexpr (RowOp::kAhead) {
            int next = code(0);
            auto fetched = op.fetch(next);
            for (int s = 0; s < steps; ++s) {
                const int e = next;
                const auto f = fetched;
                const bool v = valid;
                next = code(s + 1);
                fetched = op.fetch(next);
                op.pair(v, e, f);
            }
        } else {
            for (int s = 0; s < steps; ++s) {
                const int e = code(s);
                op.pair(valid, e);
            }
        }
        r.head += min(4 * m, cnt);
    }
    __device__ __forceinline__ void end(const ColRow& r) { op.end(r.si, r.vi); }
};

// entries from, from + 1, .. from + n - 1 (n <= kColBlock) of a row that is not
// in the list, in the list's order, followed by three empty ones
static __device__ __noinline__ void col_gather_block(const PairArgs& p, int row, int from, int n, int* ent)
{
    const float4 ic = p.ibox[2 * row], ih = p.ibox[2 * row + 1];
    __syncwarp();
    col_gather<false>(p, row, p.ccol[row], ic, ih, col_list_lim(p), ent, from, n);
    const int lane = threadIdx.x & 31;
    if (lane < 3) ent[n + lane] = p.col_none;
    __syncwarp();
}

// the rows (p.rows_split shares of each) in a fixed order
template <bool DIFFMOL, class RowOp>
__device__ __forceinline__ void col_rows64(const PairArgs& p, ColRowsShared& sh, RowOp& rop)
{
    const int split = p.rows_split;
    const int rows = p.ccstart[p.cg.ncol];
    // a refused system (another force of the group) has no whole list
    const int n_items = (*p.status & kStatusColumns) ? 0 : rows * split;
    const int warps = gridDim.x * (blockDim.x >> 5);
    const ColTest t = col_test(p);
    ColOp64<RowOp> op{rop};
    for (int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < n_items; item += warps) {
        const int row = item / split, part = item - row * split;
        const int2 re = p.rowent[row];                // first entry (< 0: not listed), entries
        const int b = (int)((long long)re.y * part / split), e = (int)((long long)re.y * (part + 1) / split);
        ColRow r;
        col_row_begin(p, t, row, r);
        op.begin(r);
        // the entries in blocks: of the list, or, for a row that is not in it,
        // gathered again (the same in the same order: the results do not
        // depend on which rows fitted)
        for (int k = b;;) {
            const int n = min(kColBlock, e - k);
            if (re.x >= 0) col_stage(p, p.clist + re.x + k, n, sh.ent);
            else col_gather_block(p, row, k, n, sh.ent);
            k += n;
            col_entries<DIFFMOL, false>(p, t, r, sh.ring, sh.ent, n, k >= e, op);
            if (k >= e) break;
        }
        op.end(r);
        __syncwarp();
    }
}

// ---------------------------------------------------------------- K9: forces
// One force component of a slot.  Up to 200 kcal/mol/A it goes
// to the finer of the slot's two sums (2^44: the rounding of a pair's share is
// a sixteenth of the other's quantum, and a few thousand such shares stay
// inside 64 bits), above that (NaN too) to the wide one.
__device__ __forceinline__ void row_add(const PairArgs& p, int slot, int c, double v)
{
    if (fabs(v) < 200.0)
        atomicAdd(p.faccj + 3 * (size_t)slot + c, (unsigned long long)__double2ll_rn(v * kScaleRowJ));
    else
        fixed_add(p.facc + 3 * (size_t)slot + c, v, p.scale, p.status);
}

// all three components, one test of their magnitudes (by the high words: 200
// there is its bit pattern, and infinities and NaN are above)
__device__ __forceinline__ void row_add3(const PairArgs& p, int slot, double x, double y, double z)
{
    const int lim = __double2hiint(200.0);
    const int hx = __double2hiint(x) & 0x7fffffff, hy = __double2hiint(y) & 0x7fffffff, hz = __double2hiint(z) & 0x7fffffff;
    if (max(hx, max(hy, hz)) < lim) {
        unsigned long long* to = p.faccj + 3 * (size_t)slot;
        atomicAdd(to, (unsigned long long)__double2ll_rn(x * kScaleRowJ));
        atomicAdd(to + 1, (unsigned long long)__double2ll_rn(y * kScaleRowJ));
        atomicAdd(to + 2, (unsigned long long)__double2ll_rn(z * kScaleRowJ));
    } else {
        row_add(p, slot, 0, x);
        row_add(p, slot, 1, y);
        row_add(p, slot, 2, z);
    }
}

template <bool COL, int NT, int P0, int S0, int P1, int S1>
struct ForceRow {
    // With a table every pair waits for its j-atom and then for its table row:
    // the next pair's j-atom is loaded meanwhile (192k atoms, both terms from
    // tables: 1337 -> 1269 us).  The other terms take the registers for a fifth
    // block instead (14,281 atoms: 169 us, with the early load 177).
    static constexpr bool kAhead = COL && (pot_table(P0) || (NT > 1 && pot_table(P1)));
    struct Fetched { double4 P; int type; };
    const PairArgs& p;
    double4 Pi;
    int4 mi;
    double fx, fy, fz;
    double el, ec, v[6];

    __device__ __forceinline__ void init()
    {
        el = ec = 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] = 0.0;
    }
    __device__ __forceinline__ void begin(int si, bool)
    {
        Pi = row_pos<COL>(p, si);
        mi = row_meta<COL>(p, si);
        fx = fy = fz = 0.0;
    }
    __device__ __forceinline__ Fetched fetch(int e) const
    {
        const int j = e & kCodeSlot;
        return {row_pos<COL>(p, j), row_type<COL>(p, j)};
    }
    __device__ __forceinline__ void pair(bool valid, int e) { pair(valid, e, fetch(e)); }
    __device__ __forceinline__ void pair(bool valid, int e, const Fetched& fe)
    {
        const int j = e & kCodeSlot;
        const double4 Pj = fe.P;
        const int tj = fe.type;
        const double dx = image_diff(Pi.x, Pj.x, p.pbc.e1x, p.pbc.e1rx);
        const double dy = image_diff(Pi.y, Pj.y, p.pbc.e2y, p.pbc.e2ry);
        const double dz = image_diff(Pi.z, Pj.z, p.pbc.e3z, p.pbc.e3rz);
        const double d2 = valid ? dnorm2(dx, dy, dz) : 1.0;
        double ft, e0, e1;
        pair_f64<NT, P0, S0, P1, S1>(p, d2, Pi.w, Pj.w, mi.y, tj, (e & kCodeMod) ? PMGPU_EXCL_MODIFIED : PMGPU_EXCL_NONE,
                                     ft, e0, e1);
        if (!valid) { ft = 0.0; e0 = 0.0; e1 = 0.0; }
        if (COL && valid) {
            // the half list: the j side's force too
            row_add3(p, j, dx * ft, dy * ft, dz * ft);
        }
        if (pot_lj_slot(P0)) el += e0; else ec += e0;
        if (NT > 1) { if (pot_lj_slot(P1)) el += e1; else ec += e1; }
        const double gx = dx * ft, gy = dy * ft, gz = dz * ft;
        fx -= gx; fy -= gy; fz -= gz;
        if (p.virial) {
            v[0] += gx * dx; v[1] += gx * dy; v[2] += gx * dz;
            v[3] += gy * dy; v[4] += gy * dz; v[5] += gz * dz;
        }
        if (p.rec_pairs && valid) {                  // diagnostic pair recording, once a pair
            const int oj = row_meta<COL>(p, j).x;
            if (COL || mi.x < oj) {
                const unsigned long long k = atomicAdd(p.rec_count, 1ull);
                if ((long long)k < p.rec_cap) {
                    p.rec_pairs[2 * k] = min(mi.x, oj);
                    p.rec_pairs[2 * k + 1] = max(mi.x, oj);
                }
            }
        }
    }
    __device__ __forceinline__ void end(int si, bool vi)
    {
        fx = row_sum(fx); fy = row_sum(fy); fz = row_sum(fz);
        const int jj = (threadIdx.x & 31) >> 3;
        if (vi && jj < 3) {
            const double v = jj == 0 ? fx : (jj == 1 ? fy : fz);
            row_add(p, si, jj, v);
        }
    }
};

// weight: a half where every pair was visited from both of its atoms
template <class Op>
__device__ __forceinline__ void force_record(const PairArgs& p, const Op& op, double weight)
{
    const double el = weight * op.el, ec = weight * op.ec;
    double v[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = weight * op.v[k];
    double acc[kERec] = {el, ec, v[0], v[1], v[2], v[1], v[3], v[4], v[2], v[4], v[5]};
    block_reduce_store<4>(acc, p.erec, p.erec_stride, blockIdx.x);
}

template <int NT, int P0, int S0, int P1, int S1>
__global__ void __launch_bounds__(128, 4) k_pair_fp64(const __grid_constant__ PairArgs p)
{
    __shared__ RowsShared sh[4];
    ForceRow<false, NT, P0, S0, P1, S1> op{p};
    op.init();
    cell_rows<false>(p, sh[threadIdx.x >> 5], op);
    force_record(p, op, 0.5);
}

// blocks an SM: with a table 4 (a fifth spills, and 192k atoms take 1334 us for
// 1329), else 5 (the pair phase waits for its own results, 49% of the issue
// slots used; 14,281 atoms: 191 -> 169 us)
template <int NT, int P0, int P1>
constexpr int kRow64Blocks = pot_table(P0) || (NT > 1 && pot_table(P1)) ? 4 : 5;

template <int NT, int P0, int S0, int P1, int S1>
__global__ void __launch_bounds__(128, kRow64Blocks<NT, P0, P1>) k_pair_fp64_col(const __grid_constant__ PairArgs p)
{
    pdl_wait();
    __shared__ ColRowsShared sh[4];
    ForceRow<true, NT, P0, S0, P1, S1> op{p};
    op.init();
    col_rows64<false>(p, sh[threadIdx.x >> 5], op);
    force_record(p, op, 1.0);
}

// ---------------------------------------------------------------- molecular virial
// Molecular virial of a cutoff force (OneAtomPair.h:174-181,
// OneAtomPairTwo.h:185-192): every pair of atoms of different molecules inside
// the cutoff adds its FP64 pair force against the minimal difference of the
// two molecules' positions (ScalarStructure::addVirial(f, diff, comDiff),
// base/ScalarStructure.cpp:90-132), and against the pair vector to the
// inter-molecular atomic virial.  A pair of one molecule adds to neither
// tensor (exclusions act only within a molecule, so none applies here).  No
// forces, no energies.
template <bool COL, int NT, int P0, int S0, int P1, int S1>
struct MolvirRow {
    static constexpr bool kAhead = false;
    const PairArgs& p;
    double4 Pi;
    int4 mi;
    double cx, cy, cz;
    double m[6], v[6];

    __device__ __forceinline__ void init()
    {
#pragma unroll
        for (int k = 0; k < 6; ++k) m[k] = v[k] = 0.0;
    }
    __device__ __forceinline__ void begin(int si, bool)
    {
        Pi = row_pos<COL>(p, si);
        mi = row_meta<COL>(p, si);
        const double* c = p.molpos + 3 * (size_t)max(mi.z, 0);      // a padding slot has no molecule
        cx = c[0]; cy = c[1]; cz = c[2];
    }
    __device__ __forceinline__ void pair(bool valid, int e)
    {
        const int j = e & kCodeSlot;
        const double4 Pj = row_pos<COL>(p, j);
        const int4 mj = row_meta<COL>(p, j);
        const double dx = image_diff(Pi.x, Pj.x, p.pbc.e1x, p.pbc.e1rx);
        const double dy = image_diff(Pi.y, Pj.y, p.pbc.e2y, p.pbc.e2ry);
        const double dz = image_diff(Pi.z, Pj.z, p.pbc.e3z, p.pbc.e3rz);
        const double d2 = valid ? dnorm2(dx, dy, dz) : 1.0;
        double ft, e0, e1;
        pair_f64<NT, P0, S0, P1, S1>(p, d2, Pi.w, Pj.w, mi.y, mj.y, PMGPU_EXCL_NONE, ft, e0, e1);
        if (!valid) ft = 0.0;
        const double gx = dx * ft, gy = dy * ft, gz = dz * ft;
        const double* c = p.molpos + 3 * (size_t)max(mj.z, 0);
        double ux, uy, uz;
        pbc_min_diff(p.pbc, cx, cy, cz, c[0], c[1], c[2], ux, uy, uz);
        m[0] += gx * ux; m[1] += gx * uy; m[2] += gx * uz; m[3] += gy * uy; m[4] += gy * uz; m[5] += gz * uz;
        v[0] += gx * dx; v[1] += gx * dy; v[2] += gx * dz; v[3] += gy * dy; v[4] += gy * dz; v[5] += gz * dz;
    }
    __device__ __forceinline__ void end(int, bool) {}
};

// weight: a half where every pair was visited from both of its atoms (cells,
// the full list), one over the half list
template <class Op>
__device__ __forceinline__ void molvir_record(const PairArgs& p, const Op& op, double weight)
{
    double acc[kMRec];
    constexpr int at[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma unroll
    for (int k = 0; k < 9; ++k) { acc[k] = weight * op.m[at[k]]; acc[9 + k] = weight * op.v[at[k]]; }
    block_reduce_store_n<4, kMRec>(acc, p.mrec, p.mrec_stride, blockIdx.x);
}

template <int NT, int P0, int S0, int P1, int S1>
__global__ void __launch_bounds__(128, 4) k_pair_molvir(const __grid_constant__ PairArgs p)
{
    __shared__ RowsShared sh[4];
    MolvirRow<false, NT, P0, S0, P1, S1> op{p};
    op.init();
    cell_rows<true>(p, sh[threadIdx.x >> 5], op);
    molvir_record(p, op, 0.5);
}

template <int NT, int P0, int S0, int P1, int S1>
__global__ void __launch_bounds__(128, 4) k_pair_molvir_col(const __grid_constant__ PairArgs p)
{
    pdl_wait();
    __shared__ ColRowsShared sh[4];
    MolvirRow<true, NT, P0, S0, P1, S1> op{p};
    op.init();
    col_rows64<true>(p, sh[threadIdx.x >> 5], op);
    molvir_record(p, op, p.col_half ? 1.0 : 0.5);
}
