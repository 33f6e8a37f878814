// pm_pair.cu -- K2 over cell clusters: launches of the mixed-precision pair
// kernels of the boxes the column layout does not take, and the ids of the
// registered combinations of terms.
#include "pm_pair_math.cuh"

namespace pm {

// ------------------------------------------------------------------ combos
struct Combo { int n, p0, s0, p1, s1; };
// The registered periodic OneAtomPair[Two] templates
// (factories/registerForceExemplarsCutoff.cpp:36-137) plus the fused
// LennardJones Coulomb -switchingFunction C2 -switchingFunction C2.  A table
// potential's own switching function is inside its table; the pair applies
// UniversalSwitchingFunction to it (combos 17-24).  Their list: PM_COMBOS.
#define PM_COMBO_ROW(_, ID, ...) {__VA_ARGS__},
static const Combo kCombos[] = {
    PM_COMBOS(PM_COMBO_ROW, 0)
};
constexpr int kNumCombos = sizeof(kCombos) / sizeof(kCombos[0]);

int pair_combo_id(int n_terms, const int* pot, const int* sw)
{
    // a table term's sw is the tabulated switching function
    const int s0 = pot_table(pot[0]) ? SUN : sw[0];
    const int s1 = n_terms > 1 && pot_table(pot[1]) ? SUN : (n_terms > 1 ? sw[1] : SUN);
    for (int k = 0; k < kNumCombos; ++k) {
        const Combo& c = kCombos[k];
        if (c.n != n_terms) continue;
        if (c.p0 == pot[0] && c.s0 == s0 && (n_terms == 1 || (c.p1 == pot[1] && c.s1 == s1)))
            return k;
    }
    return -1;
}

#include "pm_pair_mixed.cuh"

// ---------------------------------------------------------------- launch
long long plist_estimate(int n_atoms, const CellGrid& g, int nh)
{
    // every i-supercluster against every cluster of its half shell, at the
    // mean cell occupancy plus one partial cluster, with 50% slack for uneven
    // cells
    double per_cell = (double)n_atoms / (kCluster * (double)g.ncell) + 1.0;
    double supers = (double)n_atoms / (kCluster * kSuper) + g.ncell;
    return (long long)(1.5 * supers * (nh + 1) * per_cell) + 4096;
}

long long chunk_estimate(int n_atoms, const CellGrid& g, int nh, int chunk)
{
    return plist_estimate(n_atoms, g, nh) / chunk + (long long)n_atoms / (kCluster * kSuper) + g.ncell + 1024;
}

// one full wave of the mixed kernel (persistent warps take chunks of work)
template <int NT, int P0, int S0, int P1, int S1, bool WRAP>
static int run_mixed_w(const PairArgs& a, cudaStream_t s, long long* launches)
{
    static int sms = 0, per_sm = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pair_mixed<NT, P0, S0, P1, S1, WRAP>, 128, 0);
        if (sms <= 0) sms = 148;
        if (per_sm <= 0) per_sm = 1;
    }
    // a tuned number of resident blocks per SM (fewer leave room for the PME
    // kernels running beside it), else the occupancy limit
    const int bps = a.blocks_per_sm > 0 ? std::min(per_sm, a.blocks_per_sm) : per_sm;
    const int blocks = sms * bps;
    launch_pdl(k_pair_mixed<NT, P0, S0, P1, S1, WRAP>, blocks, 128, 0, s, a);
    *launches += 1;
    return (int)cudaGetLastError();
}

template <int NT, int P0, int S0, int P1, int S1>
static int run_mixed(const PairArgs& a, cudaStream_t s, long long* launches)
{
    return a.wrap ? run_mixed_w<NT, P0, S0, P1, S1, true>(a, s, launches)
                  : run_mixed_w<NT, P0, S0, P1, S1, false>(a, s, launches);
}

int launch_cluster_list(const PairArgs& a, cudaStream_t s, long long* launches)
{
    // one warp per cell and block of 32 half-shell cells
    long long warps = (long long)a.grid.ncell * ((a.nh + 1 + 31) / 32);
    int lb = (int)((warps + 3) / 4);
    launch_pdl(k_cluster_list, lb > 0 ? lb : 1, 128, 0, s, a);
    *launches += 1;
    return (int)cudaGetLastError();
}

int launch_pair_mixed(const PairArgs& a, int combo, cudaStream_t s, long long* launches)
{
    PM_COMBO_SWITCH(PM_COMBO_RETURN, run_mixed)
}

int launch_near_energy(const PairArgs& a, int combo, int n_atoms, cudaStream_t s, long long* launches)
{
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    // about 26 near pairs per atom in water, one per thread; at most one
    // resident wave (16 blocks per SM; the kernel is grid-stride)
    long long want = (30LL * n_atoms + 127) / 128;
    const int blocks = (int)std::max(1LL, std::min<long long>(want, 16LL * sms));
    PM_COMBO_SWITCH(PM_COMBO_LAUNCH, k_near_energy)
    *launches += 1;
    return (int)cudaGetLastError();
}

}  // namespace pm
