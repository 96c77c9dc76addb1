// noalloc.cu -- APE smearing in place on a caller-owned device field, without allocating.
//
// Who this is for: programs that hold their gauge field in device memory they got from somewhere
// else and may not call cudaMalloc themselves -- e.g. a host program whose device memory is handed
// out by another component (a framework's memory pool, or a fixed per-process budget that must
// account for every byte), or a steady-state measurement loop that must not pay the implicit
// device-wide synchronisation of cudaMalloc/cudaFree.  Such a caller cannot create a su2g handle
// (su2g_create allocates the field, the reduction scratch and a pinned result buffer), so this
// entry point works directly on the caller's buffer.
//
// A Jacobi smearing step reads the old field while it writes the new one, so it needs room for a
// second field.  That room is the file-scope array g_noalloc_scratch below: kNoAllocMaxSites
// sites of FP64 links (48 MiB).  Every GPU that loads this library reserves it for the lifetime
// of the process.  All calls share it; calls that overlap on the GPU (different streams, or
// different host threads without ordering) race on it and must not be issued.
#include <mutex>

#include "ape.cuh"
#include "internal.cuh"

using namespace su2g;

namespace {

// Largest lattice (sites) the static scratch holds: 393216 sites x 4 links x 4 doubles = 48 MiB.
// 24^4 = 331776 sites fits; 26^4 = 456976 does not.
constexpr long long kNoAllocMaxSites = 393216;

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocMaxSites * 16];

constexpr int kMaxDevices = 64;
std::mutex g_setup_lock;
void* g_scratch_addr[kMaxDevices] = {nullptr};

// Device address of g_noalloc_scratch on the current device.  In host code the array's name is
// only a host-side stand-in, so the address is looked up once per device (with that device
// current) and cached; a kernel is always given this looked-up address.  The cache lives as long
// as the process: after cudaDeviceReset the module is loaded again and the array may move, so a
// program that resets a device must not call this entry point afterwards (restart the process).
int scratch_address(int dev, void** out)
{
    if (dev < 0 || dev >= kMaxDevices)
        return set_error(nullptr, SU2G_EINVAL, "su2g_ape_inplace_noalloc: device %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_setup_lock);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return set_error(nullptr, SU2G_ECUDA, "su2g_ape_inplace_noalloc: cudaGetSymbolAddress failed: %s",
                             cudaGetErrorString(e));
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return SU2G_OK;
}

// A field in the reference's host layout double[V][4][4] (site, direction, c0..c3) on the device, seen
// like a Field<double>.  A link is 32 bytes: one 256-bit access where the field starts at a 32-byte
// boundary, two 128-bit ones where the caller's pointer is only 16-byte aligned.
template <bool A32>
struct AosField {
    double2* p;
    int Vh;
    __device__ __forceinline__ Q<double> ld(int mu, int, int n) const
    {
        const double2* a = p + 2 * ((size_t)n * 4 + mu);
        if (A32) return ld_256(reinterpret_cast<const Vec4d*>(a));
        Q<double> q;
        asm("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(q.c0), "=d"(q.c1) : "l"(a));
        asm("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(q.c2), "=d"(q.c3) : "l"(a + 1));
        return q;
    }
    __device__ __forceinline__ void st(int mu, int n, const Q<double>& q) const
    {
        double2* a = p + 2 * ((size_t)n * 4 + mu);
        if (A32) {
            st_256(reinterpret_cast<Vec4d*>(a), q);
        } else {
            a[0] = make_double2(q.c0, q.c1);
            a[1] = make_double2(q.c2, q.c3);
        }
    }
};

template <bool A32>
__device__ __forceinline__ void put(const AosField<A32>& f, int mu, int, int, int n, const Q<double>& q) { f.st(mu, n, q); }
__device__ __forceinline__ void put(const Field<double>& f, int mu, int par, int h, int, const Q<double>& q)
{
    f.sth(mu, par, h, q);
}

// Own link of a site (ape_staples asks for it by half-volume index, which an AosField does not use).
template <typename F>
struct AtSite {
    F f;
    int n;
    __device__ __forceinline__ Q<double> ld(int mu, int par, int m) const { return f.ld(mu, par, m); }
    __device__ __forceinline__ Q<double> ldh(int mu, int par, int) const { return f.ld(mu, par, n); }
};

// One Jacobi step from `in` into `out`: the links of the smeared directions become Proj(U + alpha S)
// with the staples of smearing.c:42-71; with COPY the other directions are copied.  One site per thread, parities paired per warp as in the handle's kernel,
// whose staple sums these are, but for the rounding of each staple by itself (ape_staples), and launched like it: a step starts
// in the tail of the one before.
template <int MODE, bool COPY, typename In, typename Out>
__global__ void __launch_bounds__(128, MODE == SU2G_APE_ALL ? 3 : (MODE == SU2G_APE_SPATIAL ? 4 : 8)) k_ape_any(In in, Out out, Geom g, double alpha)
{
    pdl_trigger();
    Site s{};
    int par, h;
    const bool valid = site_warp_pair(g, blockIdx.x, threadIdx.x, blockDim.x, s, par, h);
    pdl_wait(h, s.n);
    if (!valid) return;
    const AtSite<In> at{in, s.n};
    Q<double> res[4];
#pragma unroll
    for (int mu = 0; mu < 4; ++mu)
        if (COPY && !ape_updates(MODE, mu)) res[mu] = in.ld(mu, par, s.n);
    ape_staples<double, MODE, true, false>(at, g, s, par, h, [&](int mu, const Q<double>& u, const Q<double>& S) {
        res[mu] = q_project(q_axpy(alpha, S, u));
    });
#pragma unroll
    for (int mu = 0; mu < 4; ++mu)
        if (COPY || ape_updates(MODE, mu)) put(out, mu, par, h, s.n, res[mu]);
}

// Checkerboarded field with its smeared directions in one buffer and the others in another.
FieldCA<double> checkerboard(void* base, void* fixed, const Geom& g, int mode)
{
    void* dirs[4];
    for (int mu = 0; mu < 4; ++mu) dirs[mu] = (char*)(ape_updates(mode, mu) ? base : fixed) + (size_t)mu * g.V * 32;
    return field_ca(make_field<double>(dirs, g.Vh));
}

template <bool COPY, typename In, typename Out>
void step(const In& in, const Out& out, const Geom& g, int mode, double alpha, cudaStream_t st)
{
    const int grid = (g.V + 127) / 128;
    switch (mode) {
        case SU2G_APE_ALL: launch_pdl(k_ape_any<SU2G_APE_ALL, COPY, In, Out>, grid, 128, st, in, out, g, alpha); break;
        case SU2G_APE_SPATIAL: launch_pdl(k_ape_any<SU2G_APE_SPATIAL, COPY, In, Out>, grid, 128, st, in, out, g, alpha); break;
        default: launch_pdl(k_ape_any<SU2G_APE_TEMPORAL, COPY, In, Out>, grid, 128, st, in, out, g, alpha); break;
    }
}

__global__ void __launch_bounds__(kBlock) k_copy_aos(const double2* __restrict__ src, double2* __restrict__ dst,
                                                     long long n2)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n2) dst[i] = src[i];
}

}  // namespace

extern "C" int su2g_ape_inplace_noalloc(double* links, const int32_t dims[4], int32_t ns, double alpha, int32_t mode,
                                        void* cuda_stream)
{
    if (!links || !dims) return set_error(nullptr, SU2G_EINVAL, "su2g_ape_inplace_noalloc: null argument");
    long long V = 1;
    for (int d = 0; d < 4; ++d) {
        if (dims[d] < 2 || (dims[d] & 1))
            return set_error(nullptr, SU2G_EINVAL,
                             "su2g_ape_inplace_noalloc: extent %d of direction %d must be even and >= 2", dims[d], d);
        V *= dims[d];
    }
    if (V > kNoAllocMaxSites)
        return set_error(nullptr, SU2G_EINVAL,
                         "su2g_ape_inplace_noalloc: lattice of %lld sites exceeds the static scratch of %lld sites "
                         "(48 MiB); use a su2g handle (su2g_create + su2g_ape) for larger lattices",
                         V, kNoAllocMaxSites);
    if (ns < 0 || mode < SU2G_APE_ALL || mode > SU2G_APE_TEMPORAL || !(alpha == alpha))
        return set_error(nullptr, SU2G_EINVAL, "su2g_ape_inplace_noalloc: bad argument (ns=%d, mode=%d)", ns, mode);
    if (ns == 0) return SU2G_OK;

    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return set_error(nullptr, SU2G_ECUDA, "su2g_ape_inplace_noalloc: %s", cudaGetErrorString(e));
    // The kernels access the field 16 bytes at a time (32 where its alignment allows), so it must be 16-byte
    // aligned device (or managed) memory of the current device.  Callers hand in sub-allocations of their own pools,
    // so a bad pointer is refused here instead of faulting on the GPU.  Neither check allocates.
    if (((uintptr_t)links & 15u) != 0)
        return set_error(nullptr, SU2G_EINVAL,
                         "su2g_ape_inplace_noalloc: field pointer %p is not 16-byte aligned", (void*)links);
    cudaPointerAttributes pa;
    e = cudaPointerGetAttributes(&pa, links);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_error(nullptr, SU2G_EINVAL, "su2g_ape_inplace_noalloc: cannot query pointer %p: %s", (void*)links,
                         cudaGetErrorString(e));
    }
    if ((pa.type != cudaMemoryTypeDevice && pa.type != cudaMemoryTypeManaged) ||
        (pa.type == cudaMemoryTypeDevice && pa.device != dev))
        return set_error(nullptr, SU2G_EINVAL,
                         "su2g_ape_inplace_noalloc: field pointer %p is not device memory of the current device %d",
                         (void*)links, dev);
    void* scratch = nullptr;
    int rc = scratch_address(dev, &scratch);
    if (rc) return rc;

    const Geom g = make_geom(dims);
    cudaStream_t st = (cudaStream_t)cuda_stream;
    // Levels alternate between the caller's field and the scratch.  The first is read, and the last
    // written, in the caller's layout; those between are kept in the handle's checkerboarded layout,
    // whose loads are contiguous over a warp (the site-major one touches a line per lane), and only in
    // the directions the mode changes: the others stay where the first step copied them, in the
    // scratch -- or, for a last step that reads the field and writes over the scratch, where the second
    // step copied them again.  Twenty spatial steps at 20x16x18x14 on B200: 136 us (173 us without overlapping launches), against 819 us
    // with every level site-major, one direction after another and no shared products.  A field that is
    // not 32-byte aligned keeps its own layout throughout.
    const bool a32 = ((uintptr_t)links & 31u) == 0;
    void* const base[2] = {links, scratch};
    for (int i = 0; i < ns; ++i) {
        void *src = base[i & 1], *dst = base[(i & 1) ^ 1];
        const bool first = i == 0, last = i + 1 == ns, again = i == 1 && (ns & 1);
        const AosField<true> asrc{(double2*)src, g.Vh}, adst{(double2*)dst, g.Vh};
        const FieldCA<double> csrc = checkerboard(src, last && (ns & 1) ? src : scratch, g, mode),
                            cdst = checkerboard(dst, dst, g, mode);
        if (!a32) step<true>(AosField<false>{(double2*)src, g.Vh}, AosField<false>{(double2*)dst, g.Vh}, g, mode, alpha, st);
        else if (first && last) step<true>(asrc, adst, g, mode, alpha, st);
        else if (first) step<true>(asrc, cdst, g, mode, alpha, st);
        else if (last) step<true>(csrc, adst, g, mode, alpha, st);
        else if (again) step<true>(csrc, cdst, g, mode, alpha, st);
        else step<false>(csrc, cdst, g, mode, alpha, st);
    }
    if (ns & 1) {   // the last level is in the scratch: copy it back into the caller's field
        const long long n2 = V * 8;
        k_copy_aos<<<(int)((n2 + kBlock - 1) / kBlock), kBlock, 0, st>>>((const double2*)scratch, (double2*)links, n2);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(nullptr, SU2G_ECUDA, "su2g_ape_inplace_noalloc: launch failed: %s", cudaGetErrorString(e));
    return SU2G_OK;
}
