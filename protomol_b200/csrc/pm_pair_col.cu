// pm_pair_col.cu -- K2' and K11: launches of the pair list and the
// mixed-precision pair kernels over column clusters.
#include "pm_pair_math.cuh"

namespace pm {

#include "pm_pair_mixed.cuh"
#include "pm_pair_col.cuh"

// ---------------------------------------------------------------- column path
long long col_list_estimate(int n_atoms, const ColGrid& g, double volume, double cutoff)
{
    // the 4-atom j-clusters within the cutoff plus 1.5 column sides of each
    // row, with 30% slack
    const double rho = volume > 0.0 ? n_atoms / volume : 0.0;
    const double r = cutoff + 1.5 * std::max(g.sx, g.sy);
    const double rows = (double)n_atoms / kCluster + g.ncol + 1;
    const double per = std::min(rho * (4.0 / 3.0) * 3.14159265358979 * r * r * r / 4.0, 2.0 * rows);
    return (long long)(1.3 * rows * per) + 4096;
}

// Entries per chunk of the pair kernel.  Every chunk ends with partly filled
// rings (a fifth of its pair phase idle at 36 entries, an eighth at 75), and the
// kernel ends with its last chunks (30 us each at 36 entries): the first five
// eighths of the rows get chunks for about two of every resident warp (148 SMs
// x 16), the rest (last) for about six, never more than most (six tuned chunk
// units) or a chunk's shared memory.
int col_chunk_entries(int n_atoms, const ColGrid& g, double volume, double cutoff, int most, bool last)
{
    const double rho = volume > 0.0 ? n_atoms / volume : 0.0;
    const double r = cutoff + 0.75 * std::max(g.sx, g.sy);
    const double rows = (double)n_atoms / kCluster + 0.5 * g.ncol + 1;
    const double per = std::min(rho * (4.0 / 3.0) * 3.14159265358979 * r * r * r / 4.0, 2.0 * rows);
    const double all = rows * per * 0.5, warps = 148 * 16;
    const double want = all / ((last ? 6.0 : 2.0) * warps);
    // The shortest: 32 entries from about 2,000 atoms on (with 16 the partly
    // filled rings at the chunks' ends cost more than the even end gives: with
    // three 4,500-atom boxes in flight 40.8 us an evaluation for 43.6, 24 boxes
    // of 300 to 9,000 atoms 874 us for 922), 16 below that (1,000 atoms: 22.0 us
    // for 23.5, alone 56.9 for 60.5)
    most = std::max(16, std::min(most, kColChunk));
    const int least = std::min(most, all < 8.0 * warps ? 16 : 32);
    return std::max(least, std::min(most, 2 * (int)(0.5 * std::min(want, 1e6) + 1.0)));
}

long long col_chunk_estimate(long long entries, int n_atoms, const ColGrid& g, int chunk)
{
    return entries / std::max(1, chunk) + (long long)n_atoms / kCluster + g.ncol + 1024;
}

int launch_col_list(const PairArgs& a, cudaStream_t s, long long* launches)
{
    const int blocks = std::max(1, (a.icl_cap + 3) / 4);    // one warp per i-cluster
    launch_pdl(k_col_list, blocks, 128, 0, s, a);
    *launches += 1;
    return (int)cudaGetLastError();
}

template <int NT, int P0, int S0, int P1, int S1, bool TWO, int FINE>
static int run_col_t(const PairArgs& a, cudaStream_t s, long long* launches)
{
    static int sms = 0, per_sm = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pair_col<NT, P0, S0, P1, S1, TWO, FINE>, 128, 0);
        if (sms <= 0) sms = 148;
        if (per_sm <= 0) per_sm = 1;
    }
    const int bps = a.blocks_per_sm > 0 ? std::min(per_sm, a.blocks_per_sm) : per_sm;
    launch_pdl(k_pair_col<NT, P0, S0, P1, S1, TWO, FINE>, sms * bps, 128, 0, s, a);
    *launches += 1;
    return (int)cudaGetLastError();
}

// the terms' own cutoffs differ: a pair may be inside one of them only
static bool two_cutoffs(const PairArgs& a) { return a.n_terms > 1 && a.tf[0].cut2 != a.tf[1].cut2; }

template <int NT, int P0, int S0, int P1, int S1>
static int run_col(const PairArgs& a, cudaStream_t s, long long* launches)
{
    const bool fine = a.cg.fine != 0;
    if constexpr (NT > 1)
        if (two_cutoffs(a))
            return fine ? run_col_t<NT, P0, S0, P1, S1, true, 1>(a, s, launches)
                        : run_col_t<NT, P0, S0, P1, S1, true, 0>(a, s, launches);
    return fine ? run_col_t<NT, P0, S0, P1, S1, false, 1>(a, s, launches)
                : run_col_t<NT, P0, S0, P1, S1, false, 0>(a, s, launches);
}

int launch_pair_col(const PairArgs& a, int combo, cudaStream_t s, long long* launches)
{
    PM_COMBO_SWITCH(PM_COMBO_RETURN, run_col)
}

template <int NT, int P0, int S0, int P1, int S1, bool TWO>
static int run_col_batch_t(const BatchPairArgs& b, cudaStream_t s, long long* launches)
{
    static int sms = 0, per_sm = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pair_col_batch<NT, P0, S0, P1, S1, TWO>, 128, 0);
        if (sms <= 0) sms = 148;
        if (per_sm <= 0) per_sm = 1;
    }
    k_pair_col_batch<NT, P0, S0, P1, S1, TWO><<<sms * per_sm, 128, 0, s>>>(b);
    *launches += 1;
    return (int)cudaGetLastError();
}

template <int NT, int P0, int S0, int P1, int S1>
static int run_col_batch(const BatchPairArgs& b, cudaStream_t s, long long* launches)
{
    if constexpr (NT > 1)
        if (b.two) return run_col_batch_t<NT, P0, S0, P1, S1, true>(b, s, launches);
    return run_col_batch_t<NT, P0, S0, P1, S1, false>(b, s, launches);
}

int launch_pair_col_batch(const BatchPairArgs& b, int combo, cudaStream_t s, long long* launches)
{
    if (b.n < 1 || b.n > kBatchPairMax) return (int)cudaErrorInvalidValue;
    const BatchPairArgs& a = b;
    PM_COMBO_SWITCH(PM_COMBO_RETURN, run_col_batch)
}

int launch_near_energy_col(const PairArgs& a, int combo, int n_atoms, cudaStream_t s, long long* launches)
{
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    long long want = (30LL * n_atoms + 127) / 128;
    const int blocks = (int)std::max(1LL, std::min<long long>(want, 16LL * sms));
    PM_COMBO_SWITCH(PM_COMBO_LAUNCH, k_near_energy_col)
    *launches += 1;
    return (int)cudaGetLastError();
}

}  // namespace pm
