// measure.cu -- one configuration's measurement of the meas / qtop drivers in one call.
//
// Reference flow (LGT_Code/main_meas/meas.c:93-126; LGT_Code/main_qtop/qtop.c:76-91):
//   charge:  readConfig, smearing_APE_all(ism_tc, smpar_tc), topologicalCharge
//            (qtop.c: Q after every APE_all step from N_APE_start to N_APE_finish);
//   loops:   readConfig again, smearing_APE_temporal(ismt, smpart), smearing_APE_spatial(isms,
//            smpars), measureWilsonLoop.
// Here the field is read once (by the caller) and each branch smears away from it without changing it.
// Everything is enqueued at once and the results come back with one copy.
//
// A step of a small field is shorter than its launch takes on the host.  Fields up to kMeasGraphBytes are
// therefore replayed from a captured graph once a handle has asked for the same measurement kMeasGraphCalls times in a
// row; the smearing steps stay programmatic launches in it.  Q after 24 steps, 35 loops after 50 steps on B200, us a call,
// direct and replayed: FP32 8^4 320, 295; 20x14x16x16 457, 416; FP64 8^4 325, 312; 24^4 1936, 1903.  The call that captures,
// instantiates and first launches the graph takes 360 to 430 us more (24^4: 2340; 20x14x16x16: 790), what some 11 replays
// save: a program that stops before the limit has paid nothing, any other at most twice what the calls could have cost.
// The saving being the launches' and so the same for any field, it is under 2 % from 24^4 FP64 (42 MB) on, hence the limit.
#include <algorithm>
#include <array>
#include <cmath>
#include <tuple>
#include <vector>

#include "ape.cuh"
#include "internal.cuh"

using namespace su2g;

// What the launches of a measurement depend on: its specification and the handle's buffers.
using MeasKey = std::tuple<std::vector<int32_t>, std::vector<int32_t>, std::vector<int32_t>, std::array<double, 3>,
                           std::array<int, 3>, std::array<void*, 6>, const void*>;

// The last measurement, how often it was asked for in a row, and its graph.
struct su2g_meas_graph {
    MeasKey key;
    int calls = 1;
    std::vector<int> slot;   // d_out slot of each loop
    int nres = 0;            // d_out slots to fetch
    cudaGraphExec_t exec = nullptr;
};

namespace {

int ensure_work(su2g_lattice* h)
{
    if (h->meas_work) return SU2G_OK;
    const size_t bytes = 4ull * h->g.V * h->link_bytes;
    int rc = check_cuda(h, cudaMalloc(&h->meas_work, bytes), "allocating the measurement field");
    if (!rc) rc = check_cuda(h, cudaMalloc(&h->meas_alt, bytes), "allocating the measurement field");
    if (rc) {
        cudaFree(h->meas_work);
        cudaFree(h->meas_alt);
        h->meas_work = h->meas_alt = nullptr;
    }
    return rc;
}

// A smeared field that starts as the handle's own, which is only read: a direction's first step goes
// from the handle's links into one work field, the later ones back and forth between the two.
struct Smeared {
    su2g_lattice* h;
    void *cur[4], *next[4], *spare[4];
    explicit Smeared(su2g_lattice* hh) : h(hh)
    {
        for (int mu = 0; mu < 4; ++mu) {
            const size_t off = (size_t)mu * 2 * h->g.Vh * h->link_bytes;
            cur[mu] = h->dirp[mu];
            next[mu] = (char*)h->meas_work + off;
            spare[mu] = (char*)h->meas_alt + off;
        }
    }
    int steps(int n, int mode, double alpha)
    {
        for (int i = 0; i < n; ++i) {
            const int rc = ape_step(h, cur, next, mode, alpha);
            if (rc) return rc;
            for (int mu = 0; mu < 4; ++mu) {
                if (!ape_updates(mode, mu)) continue;
                void* was = cur[mu];
                cur[mu] = next[mu];
                next[mu] = was == h->dirp[mu] ? spare[mu] : was;
            }
        }
        return SU2G_OK;
    }
};

constexpr size_t kMeasGraphBytes = 64ull << 20;
constexpr int kMeasGraphCalls = 12;

int enqueue(su2g_lattice* h, const su2g_meas_spec* sp, std::vector<int>& slot, int& nres)
{
    int rc;
    if (sp->n_q) {
        Smeared f(h);
        int done = 0;
        for (int i = 0; i < sp->n_q; ++i) {
            if ((rc = f.steps(sp->q_ape[i] - done, SU2G_APE_ALL, sp->alpha_q))) return rc;
            done = sp->q_ape[i];
            // Q and sum |q| into d_out[2i], d_out[2i + 1]
            if ((rc = qtop_enqueue(h, f.cur, 2 * i))) return rc;
        }
    }
    slot.assign(sp->n_w, 0);
    nres = 2 * sp->n_q;
    if (sp->n_w) {
        Smeared f(h);
        if ((rc = f.steps(sp->ns_t, SU2G_APE_TEMPORAL, sp->alpha_t))) return rc;
        if ((rc = f.steps(sp->ns_s, SU2G_APE_SPATIAL, sp->alpha_s))) return rc;
        if ((rc = wilson_enqueue(h, f.cur, sp->R, sp->T, sp->n_w, nres, kOutSlots - 2 - nres, slot.data()))) return rc;
        nres = 1 + *std::max_element(slot.begin(), slot.end());
    }
    return SU2G_OK;
}

MeasKey key_of(const su2g_lattice* h, const su2g_meas_spec* sp)
{
    const bool nq = sp->n_q > 0, nw = sp->n_w > 0;
    return MeasKey({sp->q_ape, sp->q_ape + sp->n_q}, {sp->R, sp->R + sp->n_w}, {sp->T, sp->T + sp->n_w},
                   {nq ? sp->alpha_q : 0.0, nw ? sp->alpha_t : 0.0, nw ? sp->alpha_s : 0.0},
                   {nw ? sp->ns_t : 0, nw ? sp->ns_s : 0, h->ape_variant},
                   {h->dirp[0], h->dirp[1], h->dirp[2], h->dirp[3], h->meas_work, h->lines}, h->partials);
}

// The graph of a measurement whose buffers are all allocated (it has run once).
int capture(su2g_lattice* h, const su2g_meas_spec* sp, su2g_meas_graph* m)
{
    int rc = check_cuda(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal), "beginning graph capture");
    if (rc) return rc;
    cudaGraph_t graph = nullptr;
    rc = enqueue(h, sp, m->slot, m->nres);
    const cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
    if (!rc) rc = check_cuda(h, e, "ending graph capture");
    if (!rc) rc = check_cuda(h, cudaGraphInstantiate(&m->exec, graph, 0), "instantiating the measurement graph");
    if (graph) cudaGraphDestroy(graph);
    if (rc) cudaGetLastError();
    return rc;
}

}  // namespace

void su2g::release_meas_graph(su2g_lattice* h)
{
    if (!h->meas) return;
    if (h->meas->exec) cudaGraphExecDestroy(h->meas->exec);
    delete h->meas;
    h->meas = nullptr;
}

extern "C" int su2g_measure(su2g_lattice* h, const su2g_meas_spec* sp, double* q, double* w)
{
    if (!h) return set_error(nullptr, SU2G_EINVAL, "su2g_measure: null handle");
    if (!sp || sp->n_q < 0 || sp->n_w < 0 || (sp->n_q && (!sp->q_ape || !q)) || (sp->n_w && (!sp->R || !sp->T || !w)))
        return set_error(h, SU2G_EINVAL, "su2g_measure: bad specification");
    if (sp->n_q == 0 && sp->n_w == 0) return SU2G_OK;
    for (int i = 0; i < sp->n_q; ++i)
        if (sp->q_ape[i] < 0 || (i && sp->q_ape[i] < sp->q_ape[i - 1]))
            return set_error(h, SU2G_EINVAL, "su2g_measure: APE step counts must be >= 0 and ascending");
    if (sp->n_w && (sp->ns_t < 0 || sp->ns_s < 0))
        return set_error(h, SU2G_EINVAL, "su2g_measure: negative smearing steps");
    if (!std::isfinite(sp->alpha_q) || !std::isfinite(sp->alpha_t) || !std::isfinite(sp->alpha_s))
        return set_error(h, SU2G_EINVAL, "su2g_measure: smearing parameter not finite");
    int rc = sp->n_w ? wilson_check(h, sp->R, sp->T, sp->n_w, "su2g_measure") : SU2G_OK;
    if (rc) return rc;
    if (2 * sp->n_q > kOutSlots - 2) return set_error(h, SU2G_EINVAL, "su2g_measure: too many charges");
    cudaSetDevice(h->device);
    if ((rc = ensure_work(h)) || (sp->n_q > 0 && (rc = ensure_lines(h)))) return rc;
    std::vector<int> slot;
    int nres = 0;
    const bool again = !h->profiling && 4ull * h->g.V * h->link_bytes <= kMeasGraphBytes && h->meas &&
                       h->meas->key == key_of(h, sp);
    if (again && h->meas->calls < kMeasGraphCalls) ++h->meas->calls;
    if (again && h->meas->calls == kMeasGraphCalls) {
        if (!h->meas->exec && (rc = capture(h, sp, h->meas))) {
            release_meas_graph(h);
            return rc;
        }
        slot = h->meas->slot;
        nres = h->meas->nres;
        if ((rc = check_cuda(h, cudaGraphLaunch(h->meas->exec, h->stream), "replaying the measurement graph"))) return rc;
    } else {
        if (!again) release_meas_graph(h);
        if ((rc = enqueue(h, sp, slot, nres))) return rc;
        if (!again) h->meas = new su2g_meas_graph{key_of(h, sp)};
    }
    if ((rc = fetch_results(h, 0, nres))) return rc;
    for (int i = 0; i < sp->n_q; ++i) q[i] = h->h_out[2 * i];
    for (int i = 0; i < sp->n_w; ++i) w[i] = h->h_out[slot[i]];
    return SU2G_OK;
}

extern "C" int su2g_measure_release(su2g_lattice* h)
{
    if (!h) return set_error(nullptr, SU2G_EINVAL, "su2g_measure_release: null handle");
    cudaSetDevice(h->device);
    cudaStreamSynchronize(h->stream);
    release_meas_graph(h);
    cudaFree(h->meas_work);
    cudaFree(h->meas_alt);
    h->meas_work = h->meas_alt = nullptr;
    return SU2G_OK;
}
