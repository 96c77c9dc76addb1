// run.cu -- the update/measure loop of one lattice.
//
// Reference: the driver loop of LGT_Code/main/qcd.c:55-60, gaugefieldUpdate (update.c:102-175)
// followed by plaquette() (plaquette.c:67-100) after every sweep.  One block is `meas_every`
// sweeps of (n_hb heatbath + n_or overrelaxation) and the plaquette, summed inside the last
// sweep's update passes.  All blocks are enqueued without returning to the caller; each
// leaves the partial sums of its plaquette and acceptance in a region of its own, and one reduction sums
// those of several blocks, so that nothing but update passes runs between one block's sweeps and
// the next's.
//
// The launches are programmatic dependent ones (k_update), each starting in the tail of the one before.
// A captured graph of a block, replayed, ran slower on B200: its nodes did not overlap in that way and
// each replay began with a full dependency (FP64 heatbath with the plaquette every sweep, us a sweep:
// 8^4 51.2 as a graph, 29.1 as passes and 23.7 as one cluster launch, chain.cu; 24^4 140 and 92; 48^4 1520 and 1290
// -- with the faster passes).
#include <algorithm>

#include "internal.cuh"

using namespace su2g;

namespace {

constexpr size_t kPlaqScratchBytes = 64u << 20;   // plaquette partials one reduction may wait for

}  // namespace

extern "C" int su2g_graph_run(su2g_lattice* h, int32_t n_blocks, int32_t meas_every, int32_t n_hb, int32_t n_or,
                              double* plaq, double* acc)
{
    if (!h) return set_error(nullptr, SU2G_EINVAL, "su2g_graph_run: null handle");
    if (n_blocks < 0 || meas_every < 1 || n_hb < 0 || n_or < 0)
        return set_error(h, SU2G_EINVAL, "su2g_graph_run: bad counts (blocks %d, every %d, hb %d, or %d)", n_blocks,
                         meas_every, n_hb, n_or);
    if (n_blocks == 0) return SU2G_OK;
    cudaSetDevice(h->device);
    const bool fused = n_hb + n_or > 0, with_acc = n_hb > 0;
    const size_t warps = sweep_warps(h), parts = 4 * warps;   // a block's: the acceptance, the plaquette's three passes
    const int group = std::max<int>(1, std::min<size_t>(kFinSlots, kPlaqScratchBytes / (parts * sizeof(DD))));
    const bool grouped = h->chain && fused && !h->profiling &&
                         (long long)group * meas_every * (n_hb + n_or) <= kChainSubSweeps;
    int rc = fused ? ensure_partial_entries(h, parts * std::min(group, (int)n_blocks)) : SU2G_OK;
    const double nupd = (double)meas_every * n_hb * 4.0 * (double)h->g.V;
    // as many blocks at a time as there are result slots: slot 2i takes block i's plaquette, 2i + 1 its acceptance
    for (int b0 = 0; b0 < n_blocks && !rc; b0 += kOutSlots / 2) {
        const int n = std::min(n_blocks - b0, kOutSlots / 2);
        for (int i = 0; i < n && !rc; ++i) {
            const int j = i % group;
            DD* part = h->partials + j * parts;
            if (!grouped) rc = sweep_enqueue(h, meas_every, n_hb, n_or, h->hb_sweeps, part, fused, with_acc);
            else if (j == 0)   // the whole group in one launch
                rc = chain_enqueue(h, std::min(group, n - i), meas_every, n_hb, n_or, h->hb_sweeps, part, parts, true, with_acc);
            if (rc) break;
            h->hb_sweeps += (uint32_t)(meas_every * n_hb);
            double* out = h->d_out + 2 * (i - j);
            if (!fused) {
                rc = plaquette_enqueue(h, h->d_out + 2 * i);
            } else if (j == group - 1 || i == n - 1) {
                rc = sweep_plaq_finalize(h, h->partials + warps, j + 1, parts, out, 2);
                if (!rc && with_acc) rc = sweep_acc_finalize(h, h->partials, j + 1, parts, out + 1, 2);
            }
        }
        if (!rc) rc = fetch_results(h, 0, 2 * n);
        for (int i = 0; i < n && !rc; ++i) {
            if (plaq) plaq[b0 + i] = h->h_out[2 * i];
            if (acc) acc[b0 + i] = with_acc ? h->h_out[2 * i + 1] / nupd : 0.0;
        }
    }
    return rc;
}

// Nothing is kept between runs; the call waits for the handle's work, as it always has.
extern "C" int su2g_graph_release(su2g_lattice* h)
{
    if (!h) return set_error(nullptr, SU2G_EINVAL, "su2g_graph_release: null handle");
    cudaSetDevice(h->device);
    cudaStreamSynchronize(h->stream);
    return SU2G_OK;
}
