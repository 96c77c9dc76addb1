// chain.cu -- whole sweeps of a small lattice in one launch.
//
// A checkerboard pass of a lattice like the reference's own test run (8^4) is one latency chain of about
// 2 us per link: read the 18 staple links from L2, form the staple, draw, store.  Launched pass by pass (k_update)
// it takes 3 us or more, most of the rest being the hand-over from one launch to the next.  Where a pass
// fits one thread-block cluster, one link per thread, the cluster walks the passes of all sweeps itself
// and its hardware barrier separates them.
//
// The links, draws and order of operations are k_update's, and so is the assignment of links to warps, whose
// plaquette and acceptance sums go to the same entries: the fields are the same to the bit (update.cuh spells the
// multiply-adds out in FP64).  FP32 leaves them to the compiler, which starts a refused link's sums elsewhere here than in
// the passes; FP32 fields being the same in a batch and in a handle, FP32 keeps to the passes.
//
// Measured, FP64, passes -> here: 20 heatbath sweeps 427-530 -> 387-409 us (8^4), 390 -> 363 us (4^4); the loop of 10 sweeps,
// plaquette and acceptance 291 -> 237 us (8^4), 243 -> 225 us (4^4); four times 1 heatbath and 4 overrelaxation sweeps 384 -> 326
// us (8^4).  The line lies at one link per thread of 128-thread CTAs: with 256 threads the heatbath's registers leave one
// warp per scheduler waiting for two, and the one SM's load queue takes the links of both (8^4 455 against 387 us; 10^4 514 us,
// as long as the passes).  A sweep at 8^4 issues in 12 % of its SMs' cycles, the FP64 pipes 10 % busy; a warp waits 2.7
// cycles per instruction for instructions, 1.5 for fixed latencies, 1.1 for loads and 1.0 for the barrier's fence.
#include <algorithm>

#include "internal.cuh"
#include "philox.cuh"
#include "update.cuh"

using namespace su2g;

namespace {

constexpr int kCluster = 16;        // CTAs (non-portable size, asked for at creation)
constexpr int kChainThreads = 128;   // per CTA

// `n_blocks` blocks of `every` sweeps of n_hb heatbath and n_or overrelaxation sub-sweeps.  Block b's sums go
// to parts + b stride: `warps` entries of the acceptance (acc 1: set, 2: added to what is there), then three fused passes of
// as many plaquette partials (with plaq).
struct ChainArgs {
    int n_blocks, every, n_hb, n_or;
    DD* parts;
    size_t stride;
    int warps, plaq, acc;
};

__device__ __forceinline__ void cluster_arrive()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait()
{
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A thread's link of one pass: its site of the pass's parity.
struct ChainLink {
    FieldCG<double> U;   // the other CTAs' stores of the pass before are read through L2
    const Geom& g;
    int h;
    bool active;
    Site s[2];
};

template <int MU, int KIND, bool PLQ>
__device__ __forceinline__ void chain_pass(const ChainLink& l, int par, const KpBeta<double>& kb, const PhiloxKeys& keys, uint32_t sweep,
                                           uint32_t replica, unsigned* status, double* acc, DD* plaq)
{
    Site s = l.s[0];
    if (par) s = l.s[1];
    KpTrial<double> early[1];
    KpAngles<double> angles;
    if (KIND == SU2G_HEATBATH) {
        early[0] = kp_trial<double>(keys, (uint32_t)s.n, sweep, (uint32_t)MU, replica, 0u);
        angles = kp_angles<double>(keys, (uint32_t)s.n, sweep, (uint32_t)MU, replica, 0u);
        kp_pin(early, angles);
    }
    cluster_wait();
    uint32_t trials = 0;
    double p = 0.0;
    if (l.active) {
        Q<double> low;
        const Q<double> A = staple_update<double, MU, PLQ ? MU : 0>(l.U, l.g, s, par, PLQ ? &low : nullptr);
        Q<double> out;
        if (KIND == SU2G_HEATBATH) {
            if (heatbath_link<double, 1>(A, kb, keys, (uint32_t)s.n, sweep, (uint32_t)MU, replica, trials, out, status, 0u, early,
                                    angles))
                l.U.sth(MU, par, l.h, hb_store(out));
        } else {
            l.U.sth(MU, par, l.h, q_project(overrelax_link<double>(A, l.U.ldh(MU, par, l.h))));
        }
        if constexpr (PLQ) p = q_mul(l.U.ldh(MU, par, l.h), low).c0;
    }
    cluster_arrive();
    // behind the arrival: nobody waits for the sums
    if (KIND == SU2G_HEATBATH && acc) *acc += warp_acceptance(trials);
    if (PLQ) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
        if (plaq && (threadIdx.x & 31) == 0) *plaq = DD{p, 0.0};
    }
}

// One sub-sweep; `last`: its passes (1, 1), (2, 1), (3, 1) also leave their plaquette partials, at plaq and
// `warps` entries on each.
template <int KIND>
__device__ __forceinline__ void chain_sweep(const ChainLink& l, const KpBeta<double>& kb, const PhiloxKeys& keys, uint32_t sweep,
                                            uint32_t replica, unsigned* status, double* acc, bool last, DD* plaq, int warps)
{
#pragma unroll 1
    for (int par = 0; par < 2; ++par) chain_pass<0, KIND, false>(l, par, kb, keys, sweep, replica, status, acc, nullptr);
    const int plain = last ? 1 : 2;   // parities without a plaquette
#pragma unroll 1
    for (int par = 0; par < plain; ++par) chain_pass<1, KIND, false>(l, par, kb, keys, sweep, replica, status, acc, nullptr);
    if (last) chain_pass<1, KIND, true>(l, 1, kb, keys, sweep, replica, status, acc, plaq);
#pragma unroll 1
    for (int par = 0; par < plain; ++par) chain_pass<2, KIND, false>(l, par, kb, keys, sweep, replica, status, acc, nullptr);
    if (last) chain_pass<2, KIND, true>(l, 1, kb, keys, sweep, replica, status, acc, plaq ? plaq + warps : nullptr);
#pragma unroll 1
    for (int par = 0; par < plain; ++par) chain_pass<3, KIND, false>(l, par, kb, keys, sweep, replica, status, acc, nullptr);
    if (last) chain_pass<3, KIND, true>(l, 1, kb, keys, sweep, replica, status, acc, plaq ? plaq + 2 * warps : nullptr);
}

__global__ void __launch_bounds__(kChainThreads, 1) k_chain(Field<double> U0, Geom g, KpBeta<double> kb, PhiloxKeys keys,
                                                            uint32_t sweep, uint32_t replica, ChainArgs a,
                                                            unsigned* __restrict__ status)
{
    pdl_trigger();
    ChainLink l{{}, g, (int)(blockIdx.x * blockDim.x + threadIdx.x), false, {}};
    for (int d = 0; d < 4; ++d) l.U.p[d] = U0.p[d];
    l.U.Vh = U0.Vh;
    l.active = l.h < g.Vh;
    const int warp = l.h >> 5;
    l.s[0] = site_of(g, 0, l.h);
    l.s[1] = site_of(g, 1, l.h);
    pdl_wait();
    cluster_arrive();
    for (int b = 0; b < a.n_blocks; ++b) {
        DD* part = a.parts + b * a.stride + warp;
        const bool sums = warp < a.warps;
        double acc = a.acc == 2 && sums ? part->s : 0.0;
        int left = a.every * (a.n_hb + a.n_or);
        for (int s = 0; s < a.every; ++s) {
#pragma unroll 1
            for (int i = 0; i < a.n_hb; ++i, ++sweep)
                chain_sweep<SU2G_HEATBATH>(l, kb, keys, sweep, replica, status, a.acc ? &acc : nullptr,
                                              --left == 0 && a.plaq, sums ? part + a.warps : nullptr, a.warps);
#pragma unroll 1
            for (int i = 0; i < a.n_or; ++i)
                chain_sweep<SU2G_OVERRELAX>(l, kb, keys, sweep, replica, status, nullptr,
                                               --left == 0 && a.plaq, sums ? part + a.warps : nullptr, a.warps);
        }
        if (a.acc && sums && (threadIdx.x & 31) == 0) *part = DD{acc, 0.0};
    }
    cluster_wait();
}

cudaLaunchConfig_t chain_config(cudaLaunchAttribute* attr, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCluster);
    cfg.blockDim = dim3(kChainThreads);
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

}  // namespace

void su2g::chain_prepare(su2g_lattice* h)
{
    h->chain = false;
    if (h->prec != SU2G_FP64 || h->g.Vh > kCluster * kChainThreads) return;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = chain_config(attr, nullptr);
    cfg.numAttrs = 1;
    int clusters = 0;
    h->chain = cudaFuncSetAttribute(k_chain, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
               cudaOccupancyMaxActiveClusters(&clusters, k_chain, &cfg) == cudaSuccess && clusters > 0;
    cudaGetLastError();   // a device without room for it takes the passes
}

int su2g::chain_enqueue(su2g_lattice* h, int n_blocks, int every, int n_hb, int n_or, uint32_t sweep0, DD* parts,
                        size_t stride, bool plaq, int acc)
{
    const ChainArgs a{n_blocks, every, n_hb, n_or, parts, stride, sweep_warps(h), plaq, acc};
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = chain_config(attr, h->stream);
    cudaLaunchKernelEx(&cfg, k_chain, make_field<double>(h->dirp, h->g.Vh), h->g, kp_beta<double>(h->beta),
                       philox_keys(h->seed), sweep0, h->replica, a, h->d_status);
    return check_cuda(h, cudaGetLastError(), "sweeps in one launch");
}
