/*
 * mcx_kernel_label.cu -- the instantiations of the usual configurations'
 * kernel for single runs (fast math, as mcx_kernel_fast.cu).
 */
#include "mcx_kernel_label.cuh"
#include "mcx_launch.h"

#include <cstring>

namespace mcxg {

cudaError_t label_upload(const mcxg_kparams* p, const float* det4, unsigned int ndet, cudaStream_t st) {
    cudaError_t e = cudaMemcpyToSymbolAsync(c_p, p, sizeof(*p), 0, cudaMemcpyHostToDevice, st);
    float h[16] = {p->maxidx.x, p->maxidx.y, p->maxidx.z, p->oneoverc0, p->twin1, p->minenergy, p->twin0, p->Rtstep,
                   p->fxscale, p->fxunit};
    const uint32_t hi[4] = {p->dimx, p->dimxy, p->nvox, p->fieldlen};
    memcpy(h + 10, hi, sizeof(hi));
    h[14] = p->outputtype == otEnergy ? 1.f : 0.f;
    if (e == cudaSuccess) {
        e = cudaMemcpyToSymbolAsync(c_h, h, sizeof(h), 0, cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess && ndet) {
        e = cudaMemcpyToSymbolAsync(c_det, det4, sizeof(float) * 4 * ndet, 0, cudaMemcpyHostToDevice, st);
    }
    return e;
}

template <int KIND, int VOL, int DET>
static void* krefl(int flags) {
    return (flags & LF_REFL) ? (void*)mcx_transport_label<KIND, VOL, DET, true> : (void*)mcx_transport_label<KIND, VOL, DET, false>;
}

/* the replays, the RF run, the precision check: records of any kind or none */
template <int KIND, int VOL>
static void* kany(int flags) {
    return (flags & LF_DET) ? krefl<KIND, VOL, DET_ANY>(flags) : krefl<KIND, VOL, DET_NONE>(flags);
}

template <int VOL>
static void* kvol(int flags) {
    const int kinds = flags >> LF_KINDS & 0xF;     /* savedetflag's bits: 2 scatterings, 4 paths, 8 momentum */
    switch (flags >> LF_RUN & 0xF) {
    case RUN_JAC:
        return kany<RUN_JAC, VOL>(flags);
    case RUN_SITE:
        return kany<RUN_SITE, VOL>(flags);
    }
    if (!(flags & LF_DET)) {
        return krefl<RUN_FWD, VOL, DET_NONE>(flags);
    }
    if (kinds == 0) {
        return krefl<RUN_FWD, VOL, DET_ID>(flags);
    }
    if (VOL == VOL_LABEL && (kinds == 4 || kinds == 6)) {
        return kinds == 4 ? krefl<RUN_FWD, VOL_LABEL, DET_P>(flags) : krefl<RUN_FWD, VOL_LABEL, DET_SP>(flags);
    }
    return krefl<RUN_FWD, VOL, DET_ANY>(flags);
}

static void* select(int flags) {
    if ((flags >> LF_RUN & 0xF) == RUN_RF) {
        return kany<RUN_RF, VOL_LABEL>(flags);
    }
    if ((flags >> LF_RUN & 0xF) == RUN_CHECK) {
        return kany<RUN_CHECK, VOL_LABEL>(flags);
    }
    return (flags & LF_MUA) ? kvol<VOL_MUA>(flags) : kvol<VOL_LABEL>(flags);
}

/* more than 48 KB of shared memory a block has to be asked for, before the occupancy as before the launch */
static cudaError_t admit(const void* f, size_t smem) {
    return smem > 48 * 1024 ? cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
}

cudaError_t label_launch(const KArgs& a, int flags, int grid, int block, size_t smem, cudaStream_t st) {
    void* f = select(flags);
    const cudaError_t e = admit(f, smem);
    void* args[] = {(void*)&a};
    return e == cudaSuccess ? cudaLaunchKernel(f, dim3(grid), dim3(block), args, smem, st) : e;
}

cudaError_t label_occupancy(int flags, int block, size_t smem, int* blocks_per_sm) {
    void* f = select(flags);
    const cudaError_t e = admit(f, smem);
    return e == cudaSuccess ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, f, block, smem) : e;
}

cudaError_t label_attributes(int flags, cudaFuncAttributes* attr) {
    return cudaFuncGetAttributes(attr, select(flags));
}

}  // namespace mcxg
