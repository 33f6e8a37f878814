// pm_pair_rows.cu -- K9, the molecular virial and K10: launches of the FP64
// (and backward-pass) pair kernels over rows of the column list or of the
// cell-sorted clusters.
#include <cmath>

#include "pm_pair_math.cuh"

#include "pm_adjoint_math.cuh"

namespace pm {

#include "pm_pair_mixed.cuh"
#include "pm_pair_col.cuh"
#include "pm_pair_rows.cuh"

// K10 over the cell list: the backward pass of a cutoff force's pair terms
// (pm_adjoint.cu's per-pair math) over K9's rows: the row atom's dE/dq~ and
// H v sums from every pair it is in ((H v)_i += F u + 2 F' (d.u) d, u = v_j -
// v_i), dE/dA and dE/dB half to each ordered type pair, the energies half from
// each side.  The LJ table gradient goes through a small per-thread cache of
// type-pair sums (a thread's row atom keeps its type, and a few type pairs
// carry most pairs), flushed to shared or global memory on eviction and at
// the end: the table's few entries would otherwise take every pair's atomics
// on the same addresses.
constexpr int kAdjSmemTypes = 32;
constexpr int kLjCache = 4;

struct LjCache {
    long long key[kLjCache];
    double a[kLjCache], b[kLjCache];
    int hits[kLjCache];
};

__device__ __forceinline__ void lj_cache_add(LjCache& c, long long key, double pa, double pb, double* tab)
{
#pragma unroll
    for (int s = 0; s < kLjCache; ++s)
        if (c.key[s] == key) { c.a[s] += pa; c.b[s] += pb; ++c.hits[s]; return; }
    // the least used place: the solvent's few type pairs stay, and a solute
    // with a type for every atom passes through the others (14,281 atoms, 894
    // types: 1.21 -> 1.10 ms; round robin sent the solvent's pairs out as well)
    int v = 0, least = c.hits[0];
#pragma unroll
    for (int s = 1; s < kLjCache; ++s)
        if (c.hits[s] < least) { v = s; least = c.hits[s]; }
#pragma unroll
    for (int s = 0; s < kLjCache; ++s)
        if (s == v) {
            if (c.key[s] >= 0) { atomicAdd(tab + c.key[s], c.a[s]); atomicAdd(tab + c.key[s] + 1, c.b[s]); }
            c.key[s] = key; c.a[s] = pa; c.b[s] = pb; c.hits[s] = 1;
        }
}

template <bool COL, typename R>
struct AdjRow {
    static constexpr bool kAhead = false;
    const PairArgs& p;
    const AdjArgs& aa;
    double* lj_tab;
    LjCache cache;
    double el, ec;
    double4 Pi;
    int4 mi;
    double vx, vy, vz;
    double dq, hx, hy, hz;

    __device__ __forceinline__ void begin(int si, bool)
    {
        Pi = row_pos<COL>(p, si);
        const int type = mi.y;
        mi = row_meta<COL>(p, si);
        if (mi.y != type)                              // another type's pairs: all places may go
#pragma unroll
            for (int s = 0; s < kLjCache; ++s) cache.hits[s] = 0;
        vx = vy = vz = 0.0;
        if (aa.v && mi.x >= 0) { const double* v = aa.v + 3 * (size_t)mi.x; vx = v[0]; vy = v[1]; vz = v[2]; }
        dq = hx = hy = hz = 0.0;
    }
    __device__ __forceinline__ void pair(bool valid, int e)
    {
        const int j = e & kCodeSlot;
        const double4 Pj = row_pos<COL>(p, j);
        const int4 mj = row_meta<COL>(p, j);
        const double dx = image_diff(Pi.x, Pj.x, p.pbc.e1x, p.pbc.e1rx);
        const double dy = image_diff(Pi.y, Pj.y, p.pbc.e2y, p.pbc.e2ry);
        const double dz = image_diff(Pi.z, Pj.z, p.pbc.e3z, p.pbc.e3rz);
        const double a = valid ? dnorm2(dx, dy, dz) : 1.0;
        const double4 par = aa.ljd[(size_t)mi.y * aa.n_types + mj.y];
        const int excl = (e & kCodeMod) ? PMGPU_EXCL_MODIFIED : PMGPU_EXCL_NONE;
        R F, F1, pqq, pA, pB;
        adj_pair<R>(aa, a, Pi.w, Pj.w, par, excl, valid ? 0.5 : 0.0, F, F1, pqq, pA, pB, el, ec);
        if (!valid) return;
        dq += (double)pqq * Pj.w;
        if (aa.v) {
            const double* v = aa.v + 3 * (size_t)mj.x;
            const double ux = v[0] - vx, uy = v[1] - vy, uz = v[2] - vz;
            const double du = dx * ux + dy * uy + dz * uz;
            const double fF = (double)F, t2 = 2.0 * (double)F1 * du;
            hx += fF * ux + t2 * dx; hy += fF * uy + t2 * dy; hz += fF * uz + t2 * dz;
        }
        if (aa.dlj && (pA != 0 || pB != 0))
            lj_cache_add(cache, ((long long)mi.y * aa.n_types + mj.y) * 4 + (excl == PMGPU_EXCL_MODIFIED ? 2 : 0),
                         0.5 * (double)pA, 0.5 * (double)pB, lj_tab);
    }
    __device__ __forceinline__ void end(int, bool vi)
    {
        dq = row_sum(dq);
        if (aa.v) { hx = row_sum(hx); hy = row_sum(hy); hz = row_sum(hz); }
        const int jj = (threadIdx.x & 31) >> 3;
        if (!vi) return;
        if (jj == 3) {
            if (aa.dq && dq != 0.0) atomicAdd(aa.dq + mi.x, dq);
        } else if (aa.hv) {
            const double h = jj == 0 ? hx : (jj == 1 ? hy : hz);
            if (h != 0.0) atomicAdd(aa.hv + 3 * (size_t)mi.x + jj, h);
        }
    }
};

template <bool COL, typename R>
__global__ void __launch_bounds__(128) k_pair_adjoint_rows(const __grid_constant__ PairArgs p,
                                                           const __grid_constant__ AdjArgs aa)
{
    __shared__ RowsShared sh_cells[COL ? 1 : 4];
    __shared__ ColRowsShared sh_cols[COL ? 4 : 1];
    __shared__ double s_lj[kAdjSmemTypes * kAdjSmemTypes * 4];
    const bool lj_smem = aa.dlj && aa.n_types <= kAdjSmemTypes;
    if (lj_smem)
        for (int k = threadIdx.x; k < aa.n_types * aa.n_types * 4; k += blockDim.x) s_lj[k] = 0.0;
    __syncthreads();
    AdjRow<COL, R> op{p, aa};
    op.lj_tab = lj_smem ? s_lj : aa.dlj;
    op.el = op.ec = 0.0;
#pragma unroll
    for (int k = 0; k < kLjCache; ++k) { op.cache.key[k] = -1; op.cache.a[k] = 0.0; op.cache.b[k] = 0.0; op.cache.hits[k] = 0; }
    op.mi = make_int4(-1, -1, -1, 0);
    if (COL) col_rows64<false>(p, sh_cols[COL ? threadIdx.x >> 5 : 0], op);
    else cell_rows<false>(p, sh_cells[COL ? 0 : threadIdx.x >> 5], op);
#pragma unroll
    for (int k = 0; k < kLjCache; ++k)
        if (op.cache.key[k] >= 0) {
            atomicAdd(op.lj_tab + op.cache.key[k], op.cache.a[k]);
            atomicAdd(op.lj_tab + op.cache.key[k] + 1, op.cache.b[k]);
        }
    if (aa.energy) {
        double el = op.el, ec = op.ec;
        for (int o = 16; o > 0; o >>= 1) {
            el += __shfl_xor_sync(0xffffffffu, el, o);
            ec += __shfl_xor_sync(0xffffffffu, ec, o);
        }
        if ((threadIdx.x & 31) == 0) {
            if (el != 0.0) atomicAdd(aa.energy, el);
            if (ec != 0.0) atomicAdd(aa.energy + 1, ec);
        }
    }
    if (lj_smem) {
        __syncthreads();
        for (int k = threadIdx.x; k < aa.n_types * aa.n_types * 4; k += blockDim.x)
            if (s_lj[k] != 0.0) atomicAdd(aa.dlj + k, s_lj[k]);
    }
}

int launch_pair_adjoint_rows(const PairArgs& p, const AdjArgs& a, int fp64, bool col, int blocks, cudaStream_t s,
                             long long* launches)
{
    if (col) {
        if (fp64) k_pair_adjoint_rows<true, double><<<blocks, 128, 0, s>>>(p, a);
        else k_pair_adjoint_rows<true, float><<<blocks, 128, 0, s>>>(p, a);
    } else {
        if (fp64) k_pair_adjoint_rows<false, double><<<blocks, 128, 0, s>>>(p, a);
        else k_pair_adjoint_rows<false, float><<<blocks, 128, 0, s>>>(p, a);
    }
    *launches += 1;
    return (int)cudaGetLastError();
}

// ---------------------------------------------------------------- launch
// Rows are cut into shares until every resident warp (148 SMs x 16) has about
// four, so that the last wave is a quarter of the work; a share keeps at
// least eight neighbour cells.
int rows_split(int n_atoms, const CellGrid& g, int nd)
{
    const long long rows = n_atoms / kCluster + std::min(g.ncell, n_atoms) / 2 + 1;
    const long long want = (4LL * 148 * 16 + rows - 1) / rows;
    const long long most = std::max(1, std::min(kRowsSplitMax, (nd + 1) / 8));
    return (int)std::max(1LL, std::min(want, most));
}

// blocks of four warps: one share each up to one resident wave
int pair_blocks(int n_atoms, const CellGrid& g, int nd)
{
    const long long items = ((long long)n_atoms / kCluster + std::min(g.ncell, n_atoms) + 1) * rows_split(n_atoms, g, nd);
    return (int)std::max(1LL, std::min((items + 3) / 4, 148LL * 4));
}

// Shares of a row of the FP64 row kernels over the columns.  The shares go to
// the resident warps (148 SMs x 4 x blocks_per_sm) in a fixed order, so that a share count
// just above a multiple of theirs leaves most of them idle in the last round;
// a short share spends its end on partly filled rings (about twelve entries'
// worth).  The share count of the best product is taken.
int col_rows_split(int n_atoms, const ColGrid& g, double cutoff, int blocks_per_sm)
{
    const double vol = g.lx * g.ly * g.lz, rho = vol > 0.0 ? n_atoms / vol : 0.0, r = cutoff + 3.0;
    const double rows = (double)n_atoms / kCluster + 0.5 * g.ncol + 1.0;
    const double per = std::min(rho * (4.0 / 3.0) * 3.14159265358979 * r * r * r / 8.0, rows) + 1.0;
    int best = 1;
    double top = 0.0;
    for (int s = 1; s <= 16; ++s) {
        const double x = rows * s / (148.0 * 4.0 * blocks_per_sm), len = per / s;
        const double score = x / std::ceil(x) * len / (len + 12.0);
        if (score > top) { top = score; best = s; }
    }
    return best;
}

int col_row_blocks(int n_atoms, const ColGrid& g, double cutoff, int blocks_per_sm)
{
    const long long items = ((long long)n_atoms / kCluster + g.ncol + 1) * col_rows_split(n_atoms, g, cutoff, blocks_per_sm);
    return (int)std::max(1LL, std::min((items + 3) / 4, 148LL * blocks_per_sm));
}

// (the combinations from 17 on have a table)
int fp64_col_blocks_per_sm(int combo) { return combo >= 17 ? 4 : 5; }

int launch_pair_fp64(const PairArgs& a, int combo, bool col, int blocks, cudaStream_t s, long long* launches)
{
    if (col) { PM_COMBO_SWITCH(PM_COMBO_LAUNCH, k_pair_fp64_col) }
    else { PM_COMBO_SWITCH(PM_COMBO_LAUNCH, k_pair_fp64) }
    *launches += 1;
    return (int)cudaGetLastError();
}

int launch_pair_molvir(const PairArgs& a, int combo, bool col, int blocks, cudaStream_t s, long long* launches)
{
    if (col) { PM_COMBO_SWITCH(PM_COMBO_LAUNCH, k_pair_molvir_col) }
    else { PM_COMBO_SWITCH(PM_COMBO_LAUNCH, k_pair_molvir) }
    *launches += 1;
    return (int)cudaGetLastError();
}

}  // namespace pm
