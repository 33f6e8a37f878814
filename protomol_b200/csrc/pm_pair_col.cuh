// pm_pair_col.cuh -- K2a' / K2b' / K2c', K9', K10', K11: the pair kernels over
// column clusters (included after pm_pair_mixed.cuh, whose helpers the mixed
// kernel shares).
//
// Layout (K1c, pm_cells.cu): every atom holds an unsigned 32-bit fixed-point
// coordinate of the periodic box per axis, q = round(frac((x - min) / L) 2^32).
// The int32 difference of two atoms' coordinates is then their minimal-image
// displacement in units of L / 2^32, exactly: no cell offset and no rounding
// shared by the pairs of an atom or of a cell pair enters the pair vector.
// The only roundings are the conversion of that integer to FP32 and its
// product with the FP32 hi + lo of L / 2^32 (in small boxes the product's alone:
// fixed_diff).
//
// Clusters: the atoms of one column of an x-y grid (~4 A side), sorted by z,
// cut into runs of 8; each run is a row (the i side), each half of it a 4-atom
// j-cluster.
//
// K2a' k_col_list: one warp per row lists the j-clusters whose bounding box
// comes within the cutoff (plus the FP32 guard band) of the row's box by the
// nearest image.  Boxes are center and half extent; the gap of the nearest
// centers is a bound in any box.  Two forms: the half list (the forces of both
// precisions, the molecular virial: every unordered pair of atoms once) and the
// full list (the backward pass: every ordered pair once).  In the half list a pair of columns
// belongs to the one whose offset to the other is in the positive half plane
// and, within a column, a pair of rows to the lower one; where the reach covers
// the box (an offset is no longer unique) a pair of rows r < s belongs to r
// when r + s is even, else to s.  The own row's clusters come with the sign bit
// set: only j > i of them.
//
// The pair kernels take chunks of one row's entries and alternate between two
// phases (col_entries):
//
//   test   two entries (2 x 32 candidates) per step: lane l holds row atom
//          l % 8 and candidate l / 8 of the cluster; distance in FP32, the
//          exact FP64 decision inside a cutoff's guard band and the exclusion
//          class of a pair of one molecule behind a warp vote.  Pairs inside
//          the cutoff go to the row atom's ring in shared memory.
//   pairs  the lanes of a row atom take the next pairs of its ring: the pair
//          terms run on full warps.
//
// What bounds the mixed kernel: issue slots and, at five blocks per SM, the
// latency of the pair phase's chain.  An 8 x 4 tile's pairs are 40% inside the
// cutoff; evaluated tile by tile, the terms (LJ C2 + Ewald real) at 40% of the
// lanes were two thirds of the kernel's 106 M warp instructions on the
// 14,281-atom box.  The rings fill the lanes of the pair phase, and its FP32
// arithmetic is packed two pairs to an instruction: 75 M.
// Measured against the tile-by-tile kernel, each kernel alone: 8.10 -> 6.05 ms
// for 1,000,000 atoms at 12 A, 360 -> 286 us for 61,233 at 10 A, 141 -> 138 us
// for 14,281 (where 47 us do not shrink with the cutoff: the near-pair kernel's
// 13, the launch and the unevenness of the last chunks).  Tried: a full list
// with rings and no j side (152 M instructions, 217 us: the terms run twice);
// two or four times longer chunks (within 1% from 61,233 atoms on, 5% slower at
// 14,281); short chunks taken last (132 us, but 3 to 8% slower at 20,001 and
// 61,233 atoms).

constexpr int kColRing = 64;             // ring places per row atom
// entries of one row staged in shared memory (512: with 1024 the list's blocks
// held so much of it that the next kernel's first-level cache stayed small:
// 192k atoms with tables 1755 us an evaluation, 1637 with this)
constexpr int kColStageEntries = 512;
constexpr int kColBlock = 96;            // entries of a row the FP64 kernels stage at a time
constexpr int kColChunk = 64;            // most entries of a chunk of the mixed kernels
constexpr int kColNear = 128;            // near pairs a warp queues for FP64 energies
constexpr int kCodeSlot = (1 << 27) - 1; // ring code: j (a slot, or 4 x entry + atom of the chunk) | flags
constexpr int kCodeIn0 = 1 << 28, kCodeIn1 = 1 << 29, kCodeMod = 1 << 30;

// gap of two intervals (center distance d, half extents summed h) by the
// nearest image
__device__ __forceinline__ float image_gap(float d, float len, float inv, float h)
{
    d = fmaf(-len, rintf(d * inv), d);
    return fmaxf(0.f, fabsf(d) - h);
}

// the j-clusters [lo, hi) of column c whose boxes may meet the z window
// [zlo, zhi] (within [0, L)): j-boxes are sorted by z in a column (both corners
// monotone), so the column's z index gives a start at or before each end of
// the range, and a short forward scan finds it
__device__ __forceinline__ int2 col_zrange(const PairArgs& p, const int* zi, int jb, int je, float zlo, float zhi)
{
    const float inv = kZBins / p.cg.lzf;
    // first j-cluster ending at or above zlo, from the bin edge one below
    // zlo's (the FP32 bin of zlo may round up by one)
    const int b0 = zlo <= 0.f ? 0 : max(0, min(kZBins, (int)(zlo * inv)) - 1);
    int lo = max(jb, __ldg(zi + b0));
    while (lo < je && p.jbox[2 * lo].z + p.jbox[2 * lo + 1].z < zlo) ++lo;
    // first j-cluster starting above zhi, likewise from one bin edge below
    const int b1 = max(0, min(kZBins, (int)(zhi * inv)) - 1);
    int hi = max(lo, __ldg(zi + kZBins + 1 + b1));
    while (hi < je && p.jbox[2 * hi].z - p.jbox[2 * hi + 1].z <= zhi) ++hi;
    return make_int2(lo, hi);
}

// The list of one row (one warp): the columns around its own (all of them
// where the reach covers the box), in rounds of 32, one lane per column (x-y
// gap, z window, at most two ranges of j-clusters), then the round's j-clusters
// flattened over the lanes for the box tests.  The entries (j-clusters) have a
// fixed order; those from `from` on are written to out[0 .. cap).  Returns how
// many there are in all (ALL), or at least from + cap once that many are known.
// ALL looks the lanes' columns up in shared memory, the other form by shuffles
// (the FP64 kernels leave that space to the first-level cache).
template <bool ALL>
static __device__ int col_gather(const PairArgs& p, int row, int col_i, const float4& ic, const float4& ih, float lim,
                                 int* out, int from, int cap, int4* s_part = nullptr, int* s_pre = nullptr)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const ColGrid& g = p.cg;
    const float ilx = 1.0f / g.lxf, ily = 1.0f / g.lyf, ilz = 1.0f / g.lzf;
    const int nxo = min(2 * g.rx + 1, g.ncx), nyo = min(2 * g.ry + 1, g.ncy);
    const int ncand = nxo * nyo;
    const bool half = p.col_half, plane = half && nxo == 2 * g.rx + 1 && nyo == 2 * g.ry + 1;
    const int cxi = col_i / g.ncy, cyi = col_i - cxi * g.ncy;
    int ne = 0;
    for (int k0 = 0; k0 < ncand && (ALL || ne < from + cap); k0 += 32) {
        const int k = k0 + lane;
        int4 part = make_int4(0, 0, 0, 0);            // {first, count} of up to two ranges
        if (k < ncand) {
            const int ox = k / nyo - nxo / 2, oy = k % nyo - nyo / 2;
            const bool other = ox < 0 || (ox == 0 && oy < 0);     // the other column's, in the half plane rule
            int jx = cxi + ox, jy = cyi + oy;
            jx += jx < 0 ? g.ncx : 0; jx -= jx >= g.ncx ? g.ncx : 0;
            jy += jy < 0 ? g.ncy : 0; jy -= jy >= g.ncy ? g.ncy : 0;
            const int c = jx * g.ncy + jy;
            const float gx = image_gap((jx + 0.5f) * g.sx - ic.x, g.lxf, ilx, 0.5f * g.sx + ih.x);
            const float gy = image_gap((jy + 0.5f) * g.sy - ic.y, g.lyf, ily, 0.5f * g.sy + ih.y);
            const float rem = lim - (gx * gx + gy * gy);
            const int jb = 2 * (plane && c == col_i ? row : p.ccstart[c]), je = 2 * p.ccstart[c + 1];
            if (rem >= 0.f && je > jb && !(plane && other)) {
                const int* zi = p.zidx + (size_t)c * kZIndex;
                const float w = sqrtf(rem) + ih.z + 1e-3f;
                const float lo = ic.z - w, hi = ic.z + w;
                if (__ldg(zi) < 0 || 2.f * w >= g.lzf) {          // an unsorted column, or a window as high as the box
                    part = make_int4(jb, je - jb, 0, 0);
                } else if (lo < 0.f || hi > g.lzf) {              // the window wraps: its low part, then its high one
                    const int2 a = col_zrange(p, zi, jb, je, 0.f, lo < 0.f ? hi : hi - g.lzf);
                    const int2 b = col_zrange(p, zi, jb, je, lo < 0.f ? lo + g.lzf : lo, g.lzf);
                    const int b0 = max(b.x, a.y);                 // no cluster twice
                    part = make_int4(a.x, a.y - a.x, b0, max(0, b.y - b0));
                } else {
                    const int2 a = col_zrange(p, zi, jb, je, lo, hi);
                    part = make_int4(a.x, a.y - a.x, 0, 0);
                }
            }
        }
        int incl = part.y + part.w;
        const int mine = incl;
        if constexpr (ALL) s_part[lane] = part;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += v;
        }
        if constexpr (ALL) {
            s_pre[lane + 1] = incl;
            if (lane == 0) s_pre[0] = 0;
            __syncwarp();
        }
        const int total = __shfl_sync(FULL, incl, 31);
        for (int f0 = 0; f0 < total; f0 += 32) {
            const int f = f0 + lane;
            bool take = false;
            int jc = 0;
            int u = 0;
            int4 pt = part;
            if constexpr (!ALL) {                         // owner lane: the first whose sum is above f
                int own = 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    if (__shfl_sync(FULL, incl, own + o - 1) <= min(f, total - 1)) own += o;
                u = f - __shfl_sync(FULL, incl - mine, own);
                pt.x = __shfl_sync(FULL, part.x, own);
                pt.y = __shfl_sync(FULL, part.y, own);
                pt.z = __shfl_sync(FULL, part.z, own);
            }
            if (f < total) {
                if constexpr (ALL) {
                    int lo = 0, hi = 32;                  // owner lane: s_pre[lo] <= f < s_pre[lo + 1]
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (s_pre[mid] <= f) lo = mid; else hi = mid;
                    }
                    u = f - s_pre[lo];
                    pt = s_part[lo];
                }
                jc = u < pt.y ? pt.x + u : pt.z + (u - pt.y);
                const float4 bc = __ldg(p.jbox + 2 * jc), bh = __ldg(p.jbox + 2 * jc + 1);
                const float bx = image_gap(bc.x - ic.x, g.lxf, ilx, bh.x + ih.x);
                const float by = image_gap(bc.y - ic.y, g.lyf, ily, bh.y + ih.y);
                const float bz = image_gap(bc.z - ic.z, g.lzf, ilz, bh.z + ih.z);
                take = bh.w == 0.f && bx * bx + by * by + bz * bz <= lim;
                const int rj = jc >> 1;
                if (half && !plane && rj != row) take = take && (((row + rj) & 1) == 0) == (row < rj);
                if (half && rj == row) jc |= 1 << 31;
            }
            const unsigned b = __ballot_sync(FULL, take);
            const int at = ne + __popc(b & ((1u << lane) - 1u)) - from;
            if (take && at >= 0 && at < cap) out[at] = jc;
            ne += __popc(b);
        }
        __syncwarp();                                     // s_part / s_pre are rewritten next round
    }
    return ne;
}

// box distance^2 within which a j-cluster is listed; a reused list holds the
// pairs within the cutoff plus the skin.  The FP32 boxes: every corner, center
// and difference of centers is rounded by up to 2^-24 of the edge, 6.7 such
// errors in a gap and sqrt(3) of that over the axes: 7e-7 of the edge.
__device__ __forceinline__ float col_list_lim(const PairArgs& p)
{
    const float rl = sqrtf(p.cut2f) + p.list_skin + 7e-7f * fmaxf(p.cg.lxf, fmaxf(p.cg.lyf, p.cg.lzf));
    return rl * rl * (1.0f + 8.0f * p.guard) + 1e-3f;
}

static __global__ void __launch_bounds__(128) k_col_list(const __grid_constant__ PairArgs p)
{
    pdl_wait();
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ int s_ent[4][kColStageEntries];
    __shared__ int4 s_part[4][32];
    __shared__ int s_pre[4][33];
    const int row = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    if (row >= p.icl_cap) return;                                // warp-uniform
    // a refused system leaves a mark in the list's need count, which a
    // reused list keeps (the status word starts at zero every evaluation)
    if (*p.status & kStatusColumns) {
        if (row == 0 && lane == 0) atomicMax(p.plist_need, 1);
        return;
    }
    const ColGrid& g = p.cg;
    const int rows = p.ccstart[g.ncol];
    if (row >= rows) return;
    const float4 ic = p.ibox[2 * row], ih = p.ibox[2 * row + 1];
    if (p.col_refuse && 2.f * ih.z > g.zext) {                   // too tall to prune by: the cell layout
        if (lane == 0) { atomicOr(p.status, kStatusColumns); atomicMax(p.plist_need, 1); }
        return;
    }
    const float lim = col_list_lim(p);
    const int col_i = p.ccol[row];
    const int ne = col_gather<true>(p, row, col_i, ic, ih, lim, s_ent[w], 0, kColStageEntries, s_part[w], s_pre[w]);
    if (ne == 0) {                                               // not even its own cluster: cannot be
        if (lane == 0) p.rowent[row] = make_int2(0, 0);
        return;
    }
    // equal chunks of a row, an even number of entries each; the last rows'
    // (about the last to run) are shorter, so that the kernel's end is even.
    // Only the mixed kernels take chunks.
    const int most = 8 * row < 5 * rows ? p.chunk : p.chunk_end;
    const int nch = p.col_refuse ? (ne + most - 1) / most : 0;
    int b0 = 0, b1 = 0;
    if (lane == 0) {
        // A place once counted is never given back: another row may hold a
        // later one, and would share its places with the next that asks.
        bool full;
        if (p.col_refuse) {
            b0 = atomicAdd(p.plist_count, ne);
            b1 = atomicAdd(p.chunk_count, nch);
            // (a count beyond 2^31 reads as negative)
            const bool full0 = b0 < 0 || b0 > p.plist_cap - ne, full1 = b1 < 0 || b1 > p.chunk_cap - nch;
            full = full0 || full1;
            if (full) atomicOr(p.status, kStatusListFull);
            // the list buffer is counted in int2: two entries each
            if (full0) atomicMax(p.plist_need, (int)(((unsigned)b0 + (unsigned)ne) / 2) + 1);
            if (full1) atomicMax(p.chunk_need, (int)min((unsigned)b1 + (unsigned)nch, 0x7fffffffu));
        } else {
            // the FP64 kernels take a row that did not fit without its entries
            // (the same ones, gathered again); a 64-bit count cannot come round
            const unsigned long long at = atomicAdd(p.list_next, (unsigned long long)ne), end = at + ne;
            full = end > (unsigned)p.plist_cap;
            b0 = (int)at;
            if (full) {
                atomicOr(p.status, kStatusListShort);
                atomicMax(p.list_short, end);
            }
        }
        p.rowent[row] = full ? make_int2(-1, ne) : make_int2(b0, ne);
        if (full) b0 = -1;
    }
    const int ebase = __shfl_sync(FULL, b0, 0), cbase = __shfl_sync(FULL, b1, 0);
    if (ebase < 0) return;                                       // warp-uniform
    if (ne <= kColStageEntries) {
        for (int t = lane; t < ne; t += 32) p.clist[ebase + t] = s_ent[w][t];
    } else {                                              // more than the staging holds: list again, into place
        col_gather<true>(p, row, col_i, ic, ih, lim, p.clist + ebase, 0, ne, s_part[w], s_pre[w]);
    }
    if (nch == 0) return;
    const int per = ((ne + nch - 1) / nch + 1) & ~1;
    for (int t = lane; t < nch; t += 32)
        p.chunks[cbase + t] = make_int4(row, 0, ebase + t * per, max(0, min(per, ne - t * per)));
}

// ---------------------------------------------------------------- rows
// The test phase's cutoffs: pairs up to far2 are looked at, from band2 on (and
// around the smaller of two cutoffs) their decisions are taken in FP64
struct ColTest {
    float sx, sy, sz;            // L / 2^32
    float far2, band2;
    float c0, c1;                // the terms' own cutoffs^2
    float g_lo, g_hi;
};

__device__ __forceinline__ ColTest col_test(const PairArgs& p)
{
    ColTest t;
    t.sx = p.cg.sch[0]; t.sy = p.cg.sch[1]; t.sz = p.cg.sch[2];
    t.g_lo = 1.0f - p.guard; t.g_hi = 1.0f + p.guard;
    t.far2 = p.cut2f * t.g_hi;
    t.band2 = p.cut2f * t.g_lo;
    t.c0 = p.tf[0].cut2;
    t.c1 = p.n_terms > 1 ? p.tf[1].cut2 : p.tf[0].cut2;
    return t;
}

// A row's atom of the calling lane and its ring
struct ColRow {
    int si;                      // slot
    int4 P;                      // fixed-point position, molecule
    bool vi;
    float far2;                  // the test's limit (below zero for a padding atom)
    int head, tail;              // places of its ring taken / filled (the same in its four lanes)
};

// the exact decisions of one candidate (cutoff in the guard band, exclusion
// class within a molecule, j > i in the own row of a half list); code keeps
// the flags of a pair inside
template <bool DIFFMOL, bool TWO>
__device__ __forceinline__ void col_resolve(const PairArgs& p, const ColTest& t, int si, int j, bool own, float r2,
                                            bool same, bool& in, int& code)
{
    if (!in) return;
    if (own ? j <= si : j == si) { in = false; return; }
    const int oi = p.cm[si].w, oj = p.cm[j].w;
    bool band = r2 >= t.band2;
    if (TWO) band |= r2 >= fminf(t.c0, t.c1) * t.g_lo && r2 <= fminf(t.c0, t.c1) * t.g_hi;
    if (band) {
        const double d2 = exact_d2(p, oi, oj);
        if (d2 > p.cut2d) { in = false; return; }
        if (TWO) {
            code &= ~(kCodeIn0 | kCodeIn1);
            if (!(d2 > p.td[0].cut2)) code |= kCodeIn0;
            if (!(d2 > p.td[1].cut2)) code |= kCodeIn1;
        }
    }
    if (same) {
        if (DIFFMOL) { in = false; return; }
        const int x = excl_class(p, oi, oj);
        if (x == PMGPU_EXCL_FULL) in = false;
        if (x == PMGPU_EXCL_MODIFIED) code |= kCodeMod;
    }
}

// One block of up to kColBlock entries of a row, in shared memory and followed
// by three empty ones (p.col_none, a cluster of padding atoms): tested two at
// a time; op.drain runs when a ring may overflow, and to the end after the
// last block of a chunk (last).  There is one copy of it in the loop: the pair
// phase is most of the kernel's code, and a second copy (or an unrolled loop)
// did not fit the instruction cache (271 us against 150 on the 14,281-atom box,
// 8.6 of 12.8 stall cycles per instruction waiting for instructions).
// Op::kLocal: ring codes name the entry and its atom, not the slot.
template <bool DIFFMOL, bool TWO, class Op>
__device__ __forceinline__ void col_entries(const PairArgs& p, const ColTest& t, ColRow& r, int* ring, const int* ent,
                                            int n, bool last, Op& op)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, il = lane & 7, jj = lane >> 3;
    const unsigned below = (1u << (8 * jj)) - 1u;
    const int4* base = p.cq + jj;
    int2 e = *reinterpret_cast<const int2*>(ent);
    int4 A = __ldg(base + 4 * (size_t)(e.x & 0x7fffffff)), B = __ldg(base + 4 * (size_t)(e.y & 0x7fffffff));
    int* const mine = ring + il;
    for (int k = 0;; k += 2) {
        const bool done = k >= n;
        if ((done && last) || __any_sync(FULL, r.tail - r.head > kColRing - 8)) {
            __syncwarp();
            op.drain(r, ring, done && last ? 0 : Op::kKeep);
            __syncwarp();
        }
        if (done) break;
        // the next two, while these are tested
        const int2 en = *reinterpret_cast<const int2*>(ent + k + 2);
        const int4 nA = __ldg(base + 4 * (size_t)(en.x & 0x7fffffff)), nB = __ldg(base + 4 * (size_t)(en.y & 0x7fffffff));
        const float ax = (float)(int)((unsigned)A.x - (unsigned)r.P.x) * t.sx;
        const float ay = (float)(int)((unsigned)A.y - (unsigned)r.P.y) * t.sy;
        const float az = (float)(int)((unsigned)A.z - (unsigned)r.P.z) * t.sz;
        const float bx = (float)(int)((unsigned)B.x - (unsigned)r.P.x) * t.sx;
        const float by = (float)(int)((unsigned)B.y - (unsigned)r.P.y) * t.sy;
        const float bz = (float)(int)((unsigned)B.z - (unsigned)r.P.z) * t.sz;
        const float ra = fmaf(az, az, fmaf(ay, ay, ax * ax));
        const float rb = fmaf(bz, bz, fmaf(by, by, bx * bx));
        bool inA = (A.w >= 0) & (ra <= r.far2);
        bool inB = (B.w >= 0) & (rb <= r.far2);
        const bool sameA = A.w == r.P.w, sameB = B.w == r.P.w;
        int codeA = Op::kLocal ? 4 * k + jj : 4 * (e.x & 0x7fffffff) + jj;
        int codeB = Op::kLocal ? 4 * k + jj + 4 : 4 * (e.y & 0x7fffffff) + jj;
        bool rare = (inA & (sameA | (ra >= t.band2))) | (inB & (sameB | (rb >= t.band2))) | ((e.x | e.y) < 0);
        if (TWO) {                                    // two cutoffs: which terms the pair is inside of
            codeA |= (ra <= t.c0 ? kCodeIn0 : 0) | (ra <= t.c1 ? kCodeIn1 : 0);
            codeB |= (rb <= t.c0 ? kCodeIn0 : 0) | (rb <= t.c1 ? kCodeIn1 : 0);
            const float lo = fminf(t.c0, t.c1);
            rare |= (ra >= lo * t.g_lo && ra <= lo * t.g_hi) || (rb >= lo * t.g_lo && rb <= lo * t.g_hi);
        }
        if (__any_sync(FULL, rare)) {
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int eh = h ? e.y : e.x;
                bool in = h ? inB : inA;
                int code = h ? codeB : codeA;
                col_resolve<DIFFMOL, TWO>(p, t, r.si, 4 * (eh & 0x7fffffff) + jj, eh < 0, h ? rb : ra, h ? sameB : sameA,
                                          in, code);
                if (h) { inB = in; codeB = code; } else { inA = in; codeA = code; }
            }
        }
        const unsigned mA = (__ballot_sync(FULL, inA) >> il) & 0x01010101u;
        const unsigned mB = (__ballot_sync(FULL, inB) >> il) & 0x01010101u;
        const int tb = r.tail + __popc(mA);
        if (inA) mine[((r.tail + __popc(mA & below)) & (kColRing - 1)) * kCluster] = codeA;
        if (inB) mine[((tb + __popc(mB & below)) & (kColRing - 1)) * kCluster] = codeB;
        r.tail = tb + __popc(mB);
        e = en; A = nA; B = nB;
    }
}

// the row's atom for this lane
__device__ __forceinline__ void col_row_begin(const PairArgs& p, const ColTest& t, int row, ColRow& r)
{
    r.si = kCluster * row + (threadIdx.x & 7);
    r.P = p.cq[r.si];
    r.vi = r.P.w >= 0;
    r.far2 = r.vi ? t.far2 : -1.f;
    r.head = r.tail = 0;
}

// the warp's copy of n <= kColBlock entries, followed by three empty ones
__device__ __forceinline__ void col_stage(const PairArgs& p, const int* src, int n, int* ent)
{
    __syncwarp();
    for (int k = threadIdx.x & 31; k < n + 3; k += 32) ent[k] = k < n ? __ldg(src + k) : p.col_none;
    __syncwarp();
}

// sum over the four lanes of a row atom
__device__ __forceinline__ double row_sum(double v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
}

// ---------------------------------------------------------------- packed FP32
// Two FP32 values in one 64-bit register: sm_100's packed add, multiply and FMA
// do both in one issue slot, each rounded as the scalar operation.
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float lo, float hi)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ void split(F2 a, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { return fma2(b, f2(-1.f), a); }      // one rounding, as a - b
// (a - c, b - c) x (hi + lo) of fixed-point coordinates.  fine: rounded once,
// the difference's low byte beside its upper three (a byte in a float's mantissa
// is 32768 + byte; the 32768 is taken off before), and what the rounding left
// out in rest, for r^2.  Otherwise the 32-bit difference is rounded to FP32
// first, which errs alike for all pairs of a lattice that divides the box.  Such
// errors count in small boxes: the energies of 216 waters at 24 spacings were
// off by 1.1e-5 of their sum, and fine by 1.3e-6 (on the cell layout by 2.3e-6);
// C2 forces of random configurations by 1.1e-6, and fine by 2.0e-7.  The first 15
// of the 50 instructions a step took 5% of the kernel of 1,000,000 atoms: fine
// where the reach covers the box, whose evaluations take no longer for it (216
// waters 18.6 us).
__device__ __forceinline__ F2 fixed_diff(bool fine, int a, int b, int c, float hi, float lo, F2& rest)
{
    unsigned u = (unsigned)a - (unsigned)c, v = (unsigned)b - (unsigned)c;
    if (!fine) {
        const F2 d = f2((float)(int)u, (float)(int)v);
        return fma2(d, f2(hi), mul2(d, f2(lo)));
    }
    u -= 32768u;
    v -= 32768u;
    const F2 up = f2((float)(int)(u & 0xffffff00u), (float)(int)(v & 0xffffff00u));
    const F2 low = f2(__uint_as_float(__byte_perm(u, 0x47000000u, 0x7404)),
                      __uint_as_float(__byte_perm(v, 0x47000000u, 0x7404)));
    const F2 t = fma2(low, f2(hi), mul2(up, f2(lo)));
    const F2 d = fma2(up, f2(hi), t);
    rest = add2(fma2(up, f2(hi), fma2(d, f2(-1.f), f2(0.f))), t);
    return d;
}
// r^2 of fine pair vectors to the last bit, and what its rounding left out (rem):
// the squares added largest first, so that every difference below is exact
__device__ __forceinline__ F2 fine_norm2(F2 x, F2 y, F2 z, const F2 (&rest)[3], F2& rem)
{
    float x0, x1, y0, y1, z0, z1;
    split(x, x0, x1);
    split(y, y0, y1);
    split(z, z0, z1);
    const float m0 = fmaxf(fabsf(x0), fabsf(y0)), m1 = fmaxf(fabsf(x1), fabsf(y1));
    const F2 a = f2(fmaxf(m0, fabsf(z0)), fmaxf(m1, fabsf(z1)));
    const F2 b = f2(fminf(m0, fabsf(z0)), fminf(m1, fabsf(z1)));
    const F2 c = f2(fminf(fabsf(x0), fabsf(y0)), fminf(fabsf(x1), fabsf(y1)));
    const F2 s0 = mul2(a, a), s1 = fma2(b, b, s0), s2 = fma2(c, c, s1);
    const F2 e = add2(fma2(a, a, mul2(s0, f2(-1.f))), add2(fma2(b, b, sub2(s0, s1)), fma2(c, c, sub2(s1, s2))));
    const F2 low = fma2(f2(2.f), fma2(z, rest[2], fma2(y, rest[1], mul2(x, rest[0]))), e);
    const F2 r2 = add2(s2, low);
    rem = sub2(low, sub2(r2, s2));
    return r2;
}
__device__ __forceinline__ F2 sel2(bool lo, bool hi, F2 a, F2 b)
{
    float al, ah, bl, bh;
    split(a, al, ah);
    split(b, bl, bh);
    return f2(lo ? al : bl, hi ? ah : bh);
}
__device__ __forceinline__ F2 rsqrt2(F2 x)          // rsqrt_nr of both
{
    float a, b, ya, yb;
    split(x, a, b);
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(a));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(b));
    const F2 y = f2(ya, yb);
    const F2 e = fma2(mul2(x, y), y, f2(-1.f));      // the error, negated: so is the half below
    return fma2(mul2(f2(-0.5f), y), e, y);
}
__device__ __forceinline__ F2 rcp2(F2 x)            // rcp_nr of both
{
    float a, b, ya, yb;
    split(x, a, b);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(a));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(b));
    const F2 y = f2(ya, yb);
    const F2 e = fma2(x, y, f2(-1.f));
    return fma2(mul2(f2(-1.f), y), e, y);
}
__device__ __forceinline__ F2 exp_neg2(F2 x)        // exp_neg of both
{
    float a, b, ya, yb;
    split(mul2(x, f2(-1.4426950408889634f)), a, b);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(a));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(b));
    return f2(ya, yb);
}
__device__ __forceinline__ F2 poly5_2(F2 ar)        // poly5f of both
{
    const double E1 = 0.254829592, E2 = -0.284496736, E3 = 1.421413741,
                 E4 = -1.453152027, E5 = 1.061405429, PP = 0.3275911;
    const F2 t = rcp2(fma2(f2(PM_HI(PP)), ar, fma2(f2(PM_LO(PP)), ar, f2(1.0f))));
    F2 h = add2(fma2(t, f2(PM_HI(E5)), f2(PM_HI(E4))), fma2(t, f2(PM_LO(E5)), f2(PM_LO(E4))));
    h = add2(fma2(t, h, f2(PM_HI(E3))), f2(PM_LO(E3)));
    h = add2(fma2(t, h, f2(PM_HI(E2))), f2(PM_LO(E2)));
    h = add2(fma2(t, h, f2(PM_HI(E1))), f2(PM_LO(E1)));
    return mul2(t, h);
}

// pot_f32 of two pairs; m: 1-4 pairs
template <int POT>
__device__ __forceinline__ void pot2(const PairArgs& p, const TermF& t, F2 r2, F2 rd2, F2 rinv, F2 qq, int ti, int tja,
                                     int tjb, bool ma, bool mb, F2& e, F2& f)
{
    if (POT == LJ) {
        const float4 a = __ldg((ma ? p.ljm : p.ljn) + (ti * p.n_types + tja));   // A_hi, B_hi, A_lo, B_lo
        const float4 b = __ldg((mb ? p.ljm : p.ljn) + (ti * p.n_types + tjb));
        const F2 r6 = mul2(mul2(rd2, rd2), rd2), r12 = mul2(r6, r6);
        float r6a, r6b, r12a, r12b;
        split(r6, r6a, r6b);
        split(r12, r12a, r12b);
        const F2 r6B = f2(fmaf(a.y, r6a, __fmul_rn(a.w, r6a)), fmaf(b.y, r6b, __fmul_rn(b.w, r6b)));
        const F2 r12A = f2(fmaf(a.x, r12a, __fmul_rn(a.z, r12a)), fmaf(b.x, r12b, __fmul_rn(b.z, r12b)));
        e = sub2(r12A, r6B);
        f = mul2(fma2(f2(12.0f), r12A, mul2(f2(-6.0f), r6B)), rd2);
    } else if (POT == CO) {
        e = mul2(qq, rinv);
        e = sel2(ma, mb, mul2(e, f2(p.csf)), e);
        f = mul2(e, rd2);
    } else if (pot_table(POT)) {                     // (the look-ups do not pack)
        float ra, rb, qa, qb, ea, eb, fa, fb;
        split(r2, ra, rb);
        split(qq, qa, qb);
        pot_f32<POT>(p, t, ra, 0.f, 0.f, qa, ti, tja, ma ? PMGPU_EXCL_MODIFIED : PMGPU_EXCL_NONE, ea, fa);
        pot_f32<POT>(p, t, rb, 0.f, 0.f, qb, ti, tjb, mb ? PMGPU_EXCL_MODIFIED : PMGPU_EXCL_NONE, eb, fb);
        e = f2(ea, eb);
        f = f2(fa, fb);
    } else {
        const F2 q = sel2(ma, mb, mul2(qq, f2(p.csf)), qq);
        const F2 r = mul2(r2, rinv);
        const F2 ar = fma2(f2(t.alpha), r, mul2(f2(t.alpha_lo), r));
        const F2 ex = mul2(q, exp_neg2(mul2(ar, ar)));
        e = mul2(mul2(poly5_2(ar), ex), rinv);
        f = mul2(mul2(fma2(f2(t.two_alpha_pi), ex, fma2(f2(t.two_alpha_pi_lo), ex, e)), rinv), rinv);
    }
}

// sw_f32 of two pairs applied to a term (f = f v - e d, e = e v); OUT as there,
// ina / inb: inside a Cutoff switch.  FINE: r^2 is r2 + rem (the C2 switch's
// polynomials in rc^2 - r^2 lose most of the bits of r^2: their rounding was
// 85% of the virial's error of a lattice box).
template <int SW, bool OUT, bool FINE>
__device__ __forceinline__ void switch2(const TermF& t, F2 r2, F2 rem, F2 rinv, bool ina, bool inb, F2& e, F2& f)
{
    if (SW == SUN || (SW == SCUT && !OUT)) return;
    const F2 zero = f2(0.f);
    if (SW == SCUT) {
        f = sel2(ina, inb, f, zero);
        e = sel2(ina, inb, e, zero);
        return;
    }
    float ra, rb;
    split(r2, ra, rb);
    const bool oa = OUT && ra > t.cut2, ob = OUT && rb > t.cut2;
    F2 v, d;                                         // the value, and its derivative negated
    if (SW == SC2) {
        F2 c2 = sub2(f2(t.cut2), r2), u = fma2(f2(-2.0f), r2, f2(-t.s2));
        if (FINE) {
            c2 = sub2(c2, rem);
            u = fma2(f2(-2.0f), rem, u);
        }
        const F2 c4 = mul2(c2, u);                                       // negated
        const F2 c24 = mul2(c2, c4);                                     // negated
        const F2 dd = fma2(c2, c2, c4);
        const bool ma = ra >= t.on2, mb = rb >= t.on2;
        v = sel2(ma, mb, fma2(f2(-t.s1), c24, mul2(f2(-t.s1_lo), c24)), f2(1.f));
        d = sel2(ma, mb, fma2(f2(-t.s3), dd, mul2(f2(-t.s3_lo), dd)), zero);
    } else if (SW == SC1) {
        const F2 dist = mul2(r2, rinv);
        // -(fma(-r2, c05, c15) + fma(-r2, c05_lo, c15_lo)), then 1 + dist times it
        const F2 in = add2(fma2(r2, f2(t.c1_05_3), f2(-t.c1_15_1)), fma2(r2, f2(t.c1_05_3_lo), f2(-t.c1_15_1_lo)));
        v = fma2(dist, in, f2(1.f));
        d = add2(fma2(dist, f2(-t.c1_15_3), mul2(f2(t.c1_15_1), rinv)),
                 fma2(dist, f2(-t.c1_15_3_lo), mul2(f2(t.c1_15_1_lo), rinv)));
    } else {                                         // Shift
        F2 x = fma2(r2, f2(-t.sh_a_lo), fma2(r2, f2(-t.sh_a), f2(1.f)));
        if (FINE) x = fma2(rem, f2(-t.sh_a), x);
        v = mul2(x, x);
        d = fma2(f2(-t.sh_b), x, mul2(f2(-t.sh_b_lo), x));
    }
    if (OUT) {
        v = sel2(oa, ob, zero, v);
        d = sel2(oa, ob, zero, d);
    }
    f = fma2(f, v, mul2(e, d));
    e = mul2(e, v);
}

// pair_math of two pairs of one row atom: force factors and energies, zero for an
// inactive pair
template <int NT, int P0, int S0, int P1, int S1, bool OUT, bool FINE>
__device__ __forceinline__ void pair_math2(const PairArgs& p, const JAtom& ia, const JAtom& ja, const JAtom& jb, F2 r2in,
                                           F2 rem, bool va, bool vb, int ca, int cb, F2& ft, F2& el, F2& ec)
{
    constexpr bool kMod = sw_modifies(S0) || (NT > 1 && sw_modifies(S1));
    const F2 zero = f2(0.f);
    const F2 r2 = sel2(va, vb, r2in, f2(1.f));       // keeps inactive lanes finite
    const F2 rinv = rsqrt2(r2), rd2 = mul2(rinv, rinv);
    const bool ma = ca & kCodeMod, mb = cb & kCodeMod;
    F2 qq = zero;
    if (P0 != LJ || NT > 1)
        qq = f2(fmaf(ia.p.w, ja.p.w, fmaf(ia.p.w, ja.l.w, __fmul_rn(ia.l.w, ja.p.w))),
                fmaf(ia.p.w, jb.p.w, fmaf(ia.p.w, jb.l.w, __fmul_rn(ia.l.w, jb.p.w))));
    F2 e0, f0, e1 = zero, f1 = zero;
    pot2<P0>(p, p.tf[0], r2, rd2, rinv, qq, ia.m.y, ja.m.y, jb.m.y, ma, mb, e0, f0);
    if (NT > 1) pot2<P1>(p, p.tf[1], r2, rd2, rinv, qq, ia.m.y, ja.m.y, jb.m.y, ma, mb, e1, f1);
    if (kMod) {
        switch2<S0, OUT, FINE>(p.tf[0], r2, rem, rinv, ca & kCodeIn0, cb & kCodeIn0, e0, f0);
        if (NT > 1) switch2<S1, OUT, FINE>(p.tf[1], r2, rem, rinv, ca & kCodeIn1, cb & kCodeIn1, e1, f1);
    }
    ft = sel2(va, vb, NT > 1 ? add2(f0, f1) : f0, zero);
    const F2 a = sel2(va, vb, e0, zero), b = NT > 1 ? sel2(va, vb, e1, zero) : zero;
    el = pot_lj_slot(P0) ? a : zero;
    ec = pot_lj_slot(P0) ? b : a;                    // (a second term is never Lennard-Jones)
}

// ---------------------------------------------------------------- K2b': FP32 pairs
// A warp's shared memory in the mixed kernel
struct ColShared32 {
    int ring[kColRing * kCluster];
    int ent[kColChunk + 4];
    int fj[6][4 * kColChunk];            // the chunk's j-forces: steps of 2^-11, then of 2^-34; zero between chunks
    int2 near[kColNear];
    long long acc[8];                    // sums: LJ, Coulomb, virial xx xy xz yy yz zz
};
// An FP32 value in two integers without a conversion: added to 1.5 x 2^12 it is
// rounded to steps of 2^-11, in the sum's low bits, and what is left (exact, at
// most 2^-12) to steps of 2^-34 by 1.5 x 2^-11.
constexpr float kJHigh = 6144.0f, kJLow = 7.32421875e-4f;
constexpr int kJHighBits = 0x45c00000, kJLowBits = 0x3a400000;
constexpr float kLimitJ = 2047.0f;       // a j-force this large is added in 64 bits at once

// Two pairs per lane and step, their FP32 arithmetic packed (one issue slot for
// both: the kernel is bound by issue slots, not by the FMA pipe).  i-forces
// in FP32 over a drain (over a whole chunk their error against FP64 was 2-3%
// larger), far pairs' energies and virial over the chunk (at most 64 entries:
// about 15 pairs in each half of a packed sum), then FP64 and int64 fixed
// point.  j-forces are added up over the row's atoms in shared memory, each FP32
// value whole in two 32-bit integers (each atom gets at most eight per chunk:
// 2^25 in each), and added to the atoms' int64 sums once per chunk: everything
// is independent of the chunk-to-warp assignment.  One integer of 2^-23 took
// 5.65 ms instead of 6.05 for 1,000,000 atoms (133 us instead of 138 for 14,281),
// but its step is fixed: forces of 0.008 kcal/mol/A had a relative error of 5e-5,
// with two 6.5e-7, as forces of 10 have.  Near pairs (r < 5 A) go to the
// warp's queue for K2c'; their FP32 energies and virial are left out.
// TWO: the two terms' cutoffs differ (a pair may be inside one of them only).
// FINE: the grid's fine, 0 or 1, or (2, a batch's boxes) as it comes: a test a step
// costs 3% of the kernel.
template <int NT, int P0, int S0, int P1, int S1, bool TWO, int FINE>
struct ColForce32 {
    static constexpr int kKeep = 16;     // a drain leaves rings below this (longer ones share the idle lanes)
    static constexpr bool kLocal = true;
    const PairArgs& p;
    ColShared32& sh;
    int nq;
    JAtom ia;
    F2 f[3], e[2], v[6];                 // FP32 sums, first and second pairs apart
    double fs[3];                        // the row atom's force: the drains' sums

    __device__ __forceinline__ void init()
    {
        const int lane = threadIdx.x & 31;
        if (lane < 8) sh.acc[lane] = 0;
        for (int k = lane; k < 24 * kColChunk; k += 32) (&sh.fj[0][0])[k] = 0;
        nq = 0;
    }
    __device__ __forceinline__ JAtom atom(int slot) const
    {
        const int4 m = __ldg(p.cm + slot);           // charge hi, lo, type, original index
        JAtom a;
        a.p = make_float4(0.f, 0.f, 0.f, __int_as_float(m.x));
        a.l = make_float4(0.f, 0.f, 0.f, __int_as_float(m.y));
        a.m = make_int4(m.w, m.z, 0, 0);
        return a;
    }
    __device__ __forceinline__ void begin(const ColRow& r)
    {
        ia = atom(r.si);
        const F2 zero = f2(0.f);
#pragma unroll
        for (int k = 0; k < 3; ++k) fs[k] = 0.0;
        e[0] = e[1] = zero;
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] = zero;
    }
    // both halves of a sum
    static __device__ __forceinline__ double whole(F2 a)
    {
        float lo, hi;
        split(a, lo, hi);
        return (double)lo + (double)hi;
    }
    __device__ __forceinline__ int slot(int code) const
    {
        const int k = code & kCodeSlot;
        return 4 * (sh.ent[k >> 2] & 0x7fffffff) + (k & 3);
    }
    // the j-force of one pair: its two parts (t, u: sums with kJHigh, kJLow)
    __device__ __forceinline__ void add_j(int code, int slot, bool big, bool valid, const float (&v)[3],
                                          const float (&t)[3], const float (&u)[3])
    {
        if (!valid) return;
        if (!big) {
            int* to = &sh.fj[0][code & kCodeSlot];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                atomicAdd(to + c * 4 * kColChunk, __float_as_int(t[c]) - kJHighBits);
                atomicAdd(to + (3 + c) * 4 * kColChunk, __float_as_int(u[c]) - kJLowBits);
            }
        } else {
            unsigned long long* to = p.facc + 3 * (size_t)slot;
#pragma unroll
            for (int c = 0; c < 3; ++c) fixed_addf(to + c, v[c], p.status);
        }
    }
    // the pairs from places at and at + 4 of the lane's ring
    __device__ __forceinline__ void step(const ColRow& r, const int* ring, int at, bool va, bool vb)
    {
        const unsigned FULL = 0xffffffffu;
        const int lane = threadIdx.x & 31, il = lane & 7;
        const int ca = va ? ring[(at & (kColRing - 1)) * kCluster + il] : 0;
        const int cb = vb ? ring[((at + 4) & (kColRing - 1)) * kCluster + il] : 0;
        const int sa = slot(ca), sb = slot(cb);
        const JAtom ja = atom(sa), jb = atom(sb);
        const int4 A = __ldg(p.cq + sa), B = __ldg(p.cq + sb);
        const bool fine = FINE == 2 ? p.cg.fine != 0 : FINE == 1;
        F2 rest[3];
        const F2 dx = fixed_diff(fine, A.x, B.x, r.P.x, p.cg.sch[0], p.cg.scl[0], rest[0]);
        const F2 dy = fixed_diff(fine, A.y, B.y, r.P.y, p.cg.sch[1], p.cg.scl[1], rest[1]);
        const F2 dz = fixed_diff(fine, A.z, B.z, r.P.z, p.cg.sch[2], p.cg.scl[2], rest[2]);
        F2 rem = f2(0.f);
        const F2 r2 = fine ? fine_norm2(dx, dy, dz, rest, rem) : fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
        float ra, rb;
        split(r2, ra, rb);
        F2 ft, el, ec;
        pair_math2<NT, P0, S0, P1, S1, TWO, FINE != 0>(p, ia, ja, jb, r2, rem, va, vb, ca, cb, ft, el, ec);
        const F2 x = mul2(dx, ft), y = mul2(dy, ft), z = mul2(dz, ft);
        f[0] = sub2(f[0], x); f[1] = sub2(f[1], y); f[2] = sub2(f[2], z);
        float ga[3], gb[3], ta[3], tb[3], ua[3], ub[3];
        const F2 g[3] = {x, y, z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            split(g[c], ga[c], gb[c]);
            const F2 t = add2(g[c], f2(kJHigh));
            split(t, ta[c], tb[c]);
            split(add2(sub2(g[c], add2(t, f2(-kJHigh))), f2(kJLow)), ua[c], ub[c]);
        }
        // (not below the limit, and not NaN)
        const bool ba = !(fabsf(ga[0]) + fabsf(ga[1]) + fabsf(ga[2]) < kLimitJ);
        const bool bb = !(fabsf(gb[0]) + fabsf(gb[1]) + fabsf(gb[2]) < kLimitJ);
        add_j(ca, sa, ba, va, ga, ta, ua);
        add_j(cb, sb, bb, vb, gb, tb, ub);
        const bool na = va && ra < p.near2, nb = vb && rb < p.near2;           // near2 = 0: none
        if (__any_sync(FULL, na || nb)) {
            const F2 zero = f2(0.f);
            el = sel2(na, nb, zero, el);
            ec = sel2(na, nb, zero, ec);
            if (nq > kColNear - 64) { append_near(p, sh.near, nq, lane); nq = 0; }
            const unsigned wa = __ballot_sync(FULL, na), wb = __ballot_sync(FULL, nb), lt = (1u << lane) - 1u;
            if (na) sh.near[nq + __popc(wa & lt)] = make_int2(ia.m.x, ja.m.x | (ca & kCodeMod));
            nq += __popc(wa);
            if (nb) sh.near[nq + __popc(wb & lt)] = make_int2(ia.m.x, jb.m.x | (cb & kCodeMod));
            nq += __popc(wb);
        }
        e[0] = add2(e[0], el);
        e[1] = add2(e[1], ec);
        if (p.virial) {
            const F2 w = f2(na ? 0.f : 1.f, nb ? 0.f : 1.f);                   // near pairs' in FP64
            const F2 wx = mul2(x, w), wy = mul2(y, w), wz = mul2(z, w);
            v[0] = fma2(wx, dx, v[0]);
            v[1] = fma2(wx, dy, v[1]);
            v[2] = fma2(wx, dz, v[2]);
            v[3] = fma2(wy, dy, v[3]);
            v[4] = fma2(wy, dz, v[4]);
            v[5] = fma2(wz, dz, v[5]);
        }
        if (p.rec_pairs) {                             // diagnostic pair recording
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int oj = t ? jb.m.x : ja.m.x;
                if (t ? vb : va) {
                    const unsigned long long k = atomicAdd(p.rec_count, 1ull);
                    if ((long long)k < p.rec_cap) {
                        p.rec_pairs[2 * k] = min(ia.m.x, oj);
                        p.rec_pairs[2 * k + 1] = max(ia.m.x, oj);
                    }
                }
            }
        }
    }
    __device__ __forceinline__ void drain(ColRow& r, const int* ring, int keep)
    {
        // the ring's eights, each row atom from another one on: the rings of a
        // row hold the same clusters in the same order, and the same j-atom in
        // several lanes serialises their shared-memory adds
        const int lane = threadIdx.x & 31, il = lane & 7, jj = lane >> 3;
        const int cnt = r.tail - r.head;
        int m = keep ? cnt >> 3 : (cnt + 7) >> 3;
        int steps = __reduce_max_sync(0xffffffffu, m);
        if (keep) steps = max(1, steps - 2);         // the fullest ring keeps two eights: fewer idle lanes
        m = min(m, steps);
        int b = m > 0 ? il % m : 0;
        f[0] = f[1] = f[2] = f2(0.f);
        for (int s = 0; s < steps; ++s) {
            const int at = 8 * b + jj;
            step(r, ring, r.head + at, s < m && at < cnt, s < m && at + 4 < cnt);
            b = b + 1 < m ? b + 1 : 0;
        }
        r.head += min(8 * m, cnt);
#pragma unroll
        for (int k = 0; k < 3; ++k) fs[k] += whole(f[k]);
    }
    // One chunk of a row's entries
    __device__ __forceinline__ void run(const ColTest& t, const int4& cd)
    {
        const int lane = threadIdx.x & 31;
        const int n = min(cd.w, kColChunk);
        if (n <= 0) return;
        ColRow r;
        col_row_begin(p, t, cd.x, r);
        begin(r);
        col_stage(p, p.clist + cd.z, n, sh.ent);
        col_entries<false, TWO>(p, t, r, sh.ring, sh.ent, n, true, *this);
        // the chunk's j-forces
        for (int k = lane; k < 4 * n; k += 32) {
            unsigned long long* to = p.facc + 3 * (size_t)slot(k);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int q = sh.fj[c][k], l = sh.fj[3 + c][k];
                if ((q | l) != 0) {
                    sh.fj[c][k] = sh.fj[3 + c][k] = 0;
                    // to steps of 2^-32, ties to even
                    const long long v = (long long)q * 2097152 + ((l + 1 + ((l >> 2) & 1)) >> 2);
                    atomicAdd(to + c, (unsigned long long)v);
                }
            }
        }
        end(r);
    }
    __device__ __forceinline__ void end(const ColRow& r)
    {
        const int lane = threadIdx.x & 31, jj = lane >> 3;
        const double x = row_sum(fs[0]), y = row_sum(fs[1]), z = row_sum(fs[2]);
        if (r.vi && jj < 3)
            fixed_add(p.facc + 3 * (size_t)r.si + jj, jj == 0 ? x : (jj == 1 ? y : z), kScaleMixed, p.status);
        // the eight sums over the warp, scattered: lane 4 k ends with sum k
        double t[8] = {whole(e[0]), whole(e[1]), whole(v[0]), whole(v[1]), whole(v[2]), whole(v[3]), whole(v[4]),
                       whole(v[5])};
#pragma unroll
        for (int w = 4; w > 0; w >>= 1) {
            const bool up = lane & (4 * w);
#pragma unroll
            for (int k = 0; k < w; ++k) {
                const double give = up ? t[k] : t[k + w];
                t[k] = (up ? t[k + w] : t[k]) + __shfl_xor_sync(0xffffffffu, give, 4 * w);
            }
        }
        t[0] += __shfl_xor_sync(0xffffffffu, t[0], 2);
        t[0] += __shfl_xor_sync(0xffffffffu, t[0], 1);
        bool bad = false;
        if ((lane & 3) == 0) sh.acc[lane >> 2] += fixed_of(t[0], bad);
        if (bad) atomicOr(p.status, kStatusOverflow);
        if (nq > 0) { append_near(p, sh.near, nq, lane); nq = 0; }
    }
    // the warp's sums into the system's energy words (LJ, Coulomb, virial row major)
    __device__ __forceinline__ void store()
    {
        const int lane = threadIdx.x & 31;
        __syncwarp();
        if (lane < kERec) {
            constexpr int at[kERec] = {0, 1, 2, 3, 4, 3, 5, 6, 4, 6, 7};
            int k = 0;
#pragma unroll
            for (int c = 0; c < kERec; ++c) if (lane == c) k = at[c];
            const long long v = sh.acc[k];
            if (v != 0) atomicAdd(p.efix + lane, (unsigned long long)v);
        }
        __syncwarp();
        if (lane < 8) sh.acc[lane] = 0;
        __syncwarp();
    }
};

// an incomplete list (capacity exceeded or the system refused, also when it
// was built by an earlier evaluation and is reused) runs no pair
__device__ __forceinline__ int col_chunks(const PairArgs& p, bool mark)
{
    const bool bad = (*p.status & (kStatusListFull | kStatusColumns)) || *p.plist_need != 0 || *p.chunk_need != 0;
    if (bad && mark) atomicOr(p.status, kStatusListFull);
    return bad ? 0 : min(*p.chunk_count, p.chunk_cap);
}

// Blocks per SM (measured with the j-forces in one integer): five with an Ewald
// real term (96 registers, 32 bytes spilled: 5.62 against 5.84 ms for 1,000,000
// atoms, 270 against 278 us for 61,233), four
// without (the fluid of 20,001 ions: 53 against 58 us a step with three systems
// in flight, where the fifth block keeps the others' kernels waiting); six
// spill 116 bytes and take 7.96 ms.
template <int NT, int P0, int S0, int P1, int S1, bool TWO, int FINE>
__global__ void __launch_bounds__(128, P0 == EW || P1 == EW ? 5 : 4) k_pair_col(const __grid_constant__ PairArgs p)
{
    pdl_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ ColShared32 sh[4];
    const int nchunks = col_chunks(p, blockIdx.x == 0 && threadIdx.x == 0);
    const ColTest t = col_test(p);
    ColForce32<NT, P0, S0, P1, S1, TWO, FINE> op{p, sh[w]};
    op.init();
    while (true) {
        int ch = 0;
        if (lane == 0) ch = atomicAdd(p.chunk_next, 1);
        ch = __shfl_sync(0xffffffffu, ch, 0);
        if (ch >= nchunks) break;
        op.run(t, p.chunks[ch]);
    }
    op.store();
}

// K11: the column-path pair kernels of a batch's members as one persistent
// launch over (member, chunk) work items.  Every member's list was built by
// its own K2a' launch before this one.  Each block prefix-sums the members'
// chunk counts in shared memory (a member whose list is incomplete counts
// none and is marked as K2b' marks it); a warp takes items from one counter,
// copies its member's arguments into shared memory when the member changes,
// runs the chunk (as K2b') and adds its sums to the member's energy
// words when it leaves the member.  Nothing waits on another launch: the
// graph orders this one after every member's list.
template <int NT, int P0, int S0, int P1, int S1, bool TWO>
__global__ void __launch_bounds__(128, 4) k_pair_col_batch(BatchPairArgs b)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ ColShared32 sh[4];
    __shared__ int s_pre[kBatchPairMax + 1];
    __shared__ PairArgs s_args[4];
    if (threadIdx.x == 0) {
        int t = 0;
        for (int m = 0; m < b.n; ++m) {
            s_pre[m] = t;
            t += col_chunks(b.args[m], blockIdx.x == 0);
        }
        s_pre[b.n] = t;
    }
    __syncthreads();
    const int total = s_pre[b.n];
    int cur = -1;
    const PairArgs& p = s_args[w];
    ColForce32<NT, P0, S0, P1, S1, TWO, 2> op{p, sh[w]};
    op.init();
    ColTest t;
    while (true) {
        int item = 0;
        if (lane == 0) item = atomicAdd(b.next, 1);
        item = __shfl_sync(FULL, item, 0);
        if (item >= total) break;
        int lo = 0, hi = b.n;                         // the member: s_pre[lo] <= item < s_pre[lo + 1]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_pre[mid] <= item) lo = mid; else hi = mid;
        }
        if (lo != cur) {
            if (cur >= 0) op.store();
            __syncwarp();
            const int* src = reinterpret_cast<const int*>(b.args + lo);
            int* dst = reinterpret_cast<int*>(&s_args[w]);
            for (int i = lane; i < (int)(sizeof(PairArgs) / sizeof(int)); i += 32) dst[i] = src[i];
            __syncwarp();
            t = col_test(p);
            cur = lo;
        }
        op.run(t, p.chunks[item - s_pre[lo]]);
    }
    if (cur >= 0) op.store();
}

// FP64 energies and force factor of one pair of atoms by original index: the
// FP64 kernel's arithmetic (pair_f64) on the raw positions and the exact
// minimal image (d)
template <int NT, int P0, int S0, int P1, int S1>
__device__ __forceinline__ void pair_f64_orig(const PairArgs& p, int oi, int oj, int excl, double& el, double& ec,
                                              double& ft, double (&d)[3])
{
    const double* pi = p.pos + 3 * (size_t)oi;
    const double* pj = p.pos + 3 * (size_t)oj;
    const double d2 = pbc_min_diff(p.pbc, pi[0], pi[1], pi[2], pj[0], pj[1], pj[2], d[0], d[1], d[2]);
    const double qi = p.qorig[oi], qj = p.qorig[oj];
    const int ti = p.torig[oi], tj = p.torig[oj];
    double e0, e1;
    pair_f64<NT, P0, S0, P1, S1>(p, d2, qi, qj, ti, tj, excl, ft, e0, e1);
    el = (pot_lj_slot(P0) ? e0 : 0.0) + (NT > 1 && pot_lj_slot(P1) ? e1 : 0.0);
    ec = (!pot_lj_slot(P0) ? e0 : 0.0) + (NT > 1 && !pot_lj_slot(P1) ? e1 : 0.0);
}

// K2c': the FP64 energies and virial of the near pairs K2b' listed (original
// indices), each rounded to int64 fixed point on its own
template <int NT, int P0, int S0, int P1, int S1>
__global__ void __launch_bounds__(128) k_near_energy_col(const __grid_constant__ PairArgs p)
{
    const unsigned FULL = 0xffffffffu;
    __shared__ long long s_acc[8][4];
    if (*p.status & (kStatusListFull | kStatusColumns)) return;   // block-uniform
    const int n = min(*p.near_count, p.near_cap);
    long long acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};                   // LJ, Coulomb, virial xx xy xz yy yz zz
    bool bad = false;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int2 e = p.near[k];
        double el, ec, ft, d[3];
        pair_f64_orig<NT, P0, S0, P1, S1>(p, e.x, e.y & 0x3fffffff,
                                          (e.y >> 30) ? PMGPU_EXCL_MODIFIED : PMGPU_EXCL_NONE, el, ec, ft, d);
        acc[0] += fixed_of(el, bad);
        acc[1] += fixed_of(ec, bad);
        if (p.virial) {
            const double fx = ft * d[0], fy = ft * d[1], fz = ft * d[2];
            acc[2] += fixed_of(fx * d[0], bad);
            acc[3] += fixed_of(fx * d[1], bad);
            acc[4] += fixed_of(fx * d[2], bad);
            acc[5] += fixed_of(fy * d[1], bad);
            acc[6] += fixed_of(fy * d[2], bad);
            acc[7] += fixed_of(fz * d[2], bad);
        }
    }
    if (bad) atomicOr(p.status, kStatusOverflow);
    const int w = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        if (c >= 2 && !p.virial) break;
        for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(FULL, acc[c], o);
        if ((threadIdx.x & 31) == 0) s_acc[c][w] = acc[c];
    }
    __syncthreads();
    if (threadIdx.x < kERec && (threadIdx.x < 2 || p.virial)) {
        constexpr int at[kERec] = {0, 1, 2, 3, 4, 3, 5, 6, 4, 6, 7};
        int c = 0;
#pragma unroll
        for (int k = 0; k < kERec; ++k) if (threadIdx.x == k) c = at[k];
        const long long t = s_acc[c][0] + s_acc[c][1] + s_acc[c][2] + s_acc[c][3];
        if (t != 0) atomicAdd(p.efix + threadIdx.x, (unsigned long long)t);
    }
}
