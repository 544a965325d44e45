// fwi_resident.cu -- launches of the resident kernels (fwi_resident.cuh), in a
// translation unit of their own so that they compile beside the engine.
#include "fwi_resident.cuh"

namespace fwi {

template <int FP, int MODE>
static cudaError_t prepare_mode() {
    return cudaFuncSetAttribute(resident_kernel<FP, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem);
}
template <int FP>
static cudaError_t prepare() {
    cudaError_t e = prepare_mode<FP, RES_FORWARD>();
    if (e == cudaSuccess) e = prepare_mode<FP, RES_STORED>();
    if (e == cudaSuccess) e = prepare_mode<FP, RES_BOTH>();
    return e;
}
template <int FP>
static cudaError_t launch(int mode, int ctas, cudaStream_t s, ResArgs a) {
    using G = ResGeom<FP>;
    a.fields = G::fields_at(a.f.tp);
    a.sim = G::sim_floats(a.t);
    a.mat = a.fields + a.sim * (mode == RES_BOTH ? 2 : 1);
    a.xs = (G::field_floats(a.t.tzm) + 3) / 4 * 4;
    a.zs = a.xs + 8 * a.t.tzm * a.t.sxp;
    a.iw = G::inbox_words(a.t.tzm);
    void* p[] = {&a};
    const void* k = mode == RES_FORWARD  ? reinterpret_cast<const void*>(resident_kernel<FP, RES_FORWARD>)
                    : mode == RES_STORED ? reinterpret_cast<const void*>(resident_kernel<FP, RES_STORED>)
                                         : reinterpret_cast<const void*>(resident_kernel<FP, RES_BOTH>);
    return cudaLaunchCooperativeKernel(k, dim3(ctas), dim3(kResThreads), p, G::smem(a.t, a.f.tp, mode), s);
}
template <int FP>
static ResSet set() {
    return {prepare<FP>, launch<FP>, ResGeom<FP>::smem, ResGeom<FP>::inbox_words, ResGeom<FP>::RW};
}

ResSet resident_for(int fp) {
    switch (fp) {
        case 1: return set<1>();
        case 2: return set<2>();
        case 3: return set<3>();
        case 4: return set<4>();
        case 5: return set<5>();
        default: return set<6>();
    }
}

cudaError_t resident_bounds_record(unsigned long long* v) {
    *v = 0;
#if FWI_BOUNDS_CHECK
    cudaError_t e = cudaMemcpyFromSymbol(v, g_fwi_oob, sizeof(*v));
    if (e != cudaSuccess || *v == 0) return e;
    const unsigned long long zero = 0;
    return cudaMemcpyToSymbol(g_fwi_oob, &zero, sizeof(zero));
#else
    return cudaSuccess;
#endif
}

}  // namespace fwi
