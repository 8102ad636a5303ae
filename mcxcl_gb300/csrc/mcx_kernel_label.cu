/*
 * mcx_kernel_label.cu -- the transport kernel of byte-label volumes.
 *
 * The configuration most runs have -- labels in one byte a voxel, three
 * dimensions, Henyey-Greenstein, one source, real weights, flux, fluence or
 * energy deposited from launched (not replayed) photons -- with all of that
 * fixed at compile time.  The photons, their random numbers and every
 * rounding are those of mcx_transport (mcx_kernel.cuh), whose device
 * functions it shares; what differs is what a step costs.
 *
 * The kernel is bound by issue: a warp runs the scattering and the
 * voxel-crossing block in nearly every iteration, each with about half its
 * lanes, so the instructions of an iteration are what counts.  One of the
 * cube + sphere workload's took 550 (counted by ncu) and takes 300: no tests of what is
 * fixed; nothing but deposits, label and voxel index for the lanes that
 * cross a face, and what is rare (faces of the domain, label changes,
 * time-outs, roulette) behind one test; conditions combined without
 * branches; voxel coordinates as floats; the parameters of a step in four
 * vector loads; a deposit scale per label instead of a choice of output.
 * Kernel times before and after (one GB300): cube, 1e6 photons 8.95 -> 6.0 ms; cube +
 * sphere with detectors, 1e6 14.1 -> 8.9 ms, 2e7 113 -> 77 ms; head, 1e7
 * 42.9 -> 29.9 ms.
 */
#include "mcx_kernel.cuh"
#include "mcx_launch.h"

#include <cstring>

namespace mcxg {
namespace {

constexpr int LB_BLOCK = kLabelBlock;     /* threads a block: shared-memory addresses are constants plus the lane's own */

/* The parameters a step reads, in the order in which it reads them and as
   vectors, so that four come with one load: {extents, 1/c0}, {window's end,
   roulette threshold, window's start, 1/gate}, {fixed-point scale and unit,
   dimx, dimxy}, {voxels, field length, -, -}; the last six and dimx, dimxy are
   integers. */
__constant__ float4 c_h[4];

/* which partial data a run records: nothing, paths (the default 'dp'), paths
   and scattering counts ('dsp'), or whatever its flags say */
enum { DET_NONE, DET_P, DET_SP, DET_ANY };

/* Parameter source.  Shared memory: three property rows a medium --
   {mua, mus, n, 1/mus}, {1 - g^2, 1 - g, 2g, 1 + g^2}, {1/(2g), deposit scale,
   1 where flux takes the path length itself, -} -- the launch-time states, the
   partial data, one slot for each label and kind (label 0's, a photon in a
   void voxel, which has no record, included: no update needs a test), and the
   launch angle table. */
template <int DET>
struct LabelPS {
    static constexpr bool kBatch = false;
    static constexpr bool kXMedia = false;
    static constexpr bool kCommon = true;
    __device__ __forceinline__ const mcxg_kparams& p() const { return c_p; }
    __device__ __forceinline__ const float4* det() const { return c_det; }
    __device__ __forceinline__ const float4* srcx() const { return c_srcx; }
    __device__ __forceinline__ unsigned long long media_off() const { return 0ull; }
    __device__ __forceinline__ unsigned int field_off() const { return 0u; }
    __device__ __forceinline__ unsigned int lo_plane() const { return c_p.fieldlen; }
    __device__ __forceinline__ unsigned long long vt_off() const { return 0ull; }
    __device__ __forceinline__ unsigned long long seed() const { return 0ull; }
    /* kinds of partial data */
    __device__ __forceinline__ unsigned int kinds() const {
        return DET == DET_P ? 1u : (DET == DET_SP ? 2u : SAVE_NSCAT(c_p.savedetflag) + SAVE_PPATH(c_p.savedetflag) + SAVE_MOM(c_p.savedetflag));
    }
    __device__ __forceinline__ ColdState* cold() const { return (ColdState*)mcxg_smem + threadIdx.x; }
    __device__ __forceinline__ const float4* rows() const { return mcxg_smem + LB_BLOCK * sizeof(ColdState) / sizeof(float4); }
    __device__ __forceinline__ const float4& row(unsigned int label, int k) const { return rows()[3 * label + k]; }
    __device__ __forceinline__ float4 prop(const Shared&, unsigned int i) const {
        const float4 q = row(i, 0);
        return make_float4(q.x, q.y, 0.f, q.z);
    }
    __device__ __forceinline__ float* slots() const { return (float*)(rows() + 3 * c_p.medianum); }
    __device__ __forceinline__ float& slot(unsigned int kind, unsigned int label) const {
        return slots()[(label * kinds() + kind) * LB_BLOCK + threadIdx.x];
    }
    /* record entry i: label i % maxmedia + 1 of kind i / maxmedia */
    __device__ __forceinline__ float& pp(unsigned int i) const {
        unsigned int k = 0;
        while (i >= c_p.maxmedia) {
            i -= c_p.maxmedia;
            k++;
        }
        return slot(k, i + 1u);
    }
    __device__ __forceinline__ float* tables() const {
        return slots() + (DET ? kinds() * c_p.medianum * LB_BLOCK : 0u);
    }
    __device__ __forceinline__ float invcdf(unsigned int) const { return 0.f; }
    __device__ __forceinline__ float angle(unsigned int i) const { return tables()[i]; }
};

/* the bits of a volume byte */
#define LB_DET   0x80u
#define LB_LABEL 0x7Fu

/* what a lane is doing */
enum { RUN, ENDED, FRESH, DONE };

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

/* the next word of rnd's stream as a float in [1, 2): the 23 top bits under
   the exponent 0x7F in one funnel shift */
__device__ __forceinline__ float rnd12(Rng& t) {
    unsigned long long s1 = t.a;
    const unsigned long long s0 = t.b;
    t.a = s0;
    s1 ^= s1 << 23;
    t.b = s1 ^ s0 ^ (s1 >> 18) ^ (s0 >> 5);
    return __uint_as_float(__funnelshift_r((unsigned int)t.b + (unsigned int)s0, 0x7Fu, 9));
}

/* rnd_scatlen: subtracting 1 - EPS from the float in [1, 2) rounds once, as
   adding EPS to the exact u - 1 does */
__device__ __forceinline__ float lb_scatlen(Rng& t) {
    return -__logf(__fsub_rn(rnd12(t), 1.f - K_EPS));
}

/* +-1 with the sign of x.  A direction component of +0 counts as positive:
   its face is infinitely far either way. */
__device__ __forceinline__ float sign1(float x) {
    return __uint_as_float((__float_as_uint(x) & 0x80000000u) | 0x3F800000u);
}

/* rotatevector with its roundings written out, as the compiler contracts it in
   the other instantiations: a run here and its replay there follow the same
   path to the bit */
__device__ __forceinline__ void rotate_rn(float4& v, float st, float ct, float sp, float cp) {
    const float t0 = __fmaf_rn(-v.z, v.z, 1.f);
    const float t1 = __fmul_rn(st, Mth<false>::rsqrt(t0));
    const float ix = __fmaf_rn(__fmul_rn(v.x, v.z), cp, -__fmul_rn(v.y, sp));
    const float iy = __fmaf_rn(v.x, sp, __fmul_rn(__fmul_rn(v.y, v.z), cp));
    float x = __fmaf_rn(v.x, ct, __fmul_rn(t1, ix));
    float y = __fmaf_rn(v.y, ct, __fmul_rn(t1, iy));
    float z = __fmaf_rn(v.z, ct, -__fmul_rn(__fmul_rn(t1, t0), cp));
    if (!(fabsf(v.z) < 1.f - K_EPS)) {
        x = __fmul_rn(st, cp);
        y = __fmul_rn(st, sp);
        z = (v.z > 0.f) ? ct : -ct;
    }
    const float r = Mth<false>::rsqrt(__fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x))));
    v.x = __fmul_rn(x, r);
    v.y = __fmul_rn(y, r);
    v.z = __fmul_rn(z, r);
}

/* the next reference thread that has photons: with fewer photons than
   threads, the threads from the photon count on have none */
__device__ __forceinline__ int lb_claim(const KArgs& a, unsigned int& vt) {
    vt = atomicAdd(a.vtcounter, 1u);
    return vt < c_p.nthread && (c_p.threadphoton || vt < (unsigned int)c_p.oddphoton) ? FRESH : DONE;
}

/* the reference's detector flag of a photon that leaves (exit_detflag) */
__device__ __forceinline__ unsigned int lb_exitflag(unsigned int idx1d, int fw, unsigned int m) {
    return ((idx1d == K_OUT_MAX && c_p.bc[9 + fw]) || (idx1d == K_OUT_MIN && c_p.bc[6 + fw]))
           ? K_OUT_MIN : ((m & LB_DET) << 24);
}

template <int DET, bool REFL>
__global__ void __launch_bounds__(LB_BLOCK, 4) mcx_transport_label(const KArgs a) {
    typedef Mth<false> M;
    LabelPS<DET> ps;
    Shared S;
    S.bprop = S.brecip = a.gprop;
    for (unsigned int i = threadIdx.x; i < c_p.medianum; i += LB_BLOCK) {
        const float4 q = a.gprop[i];
        const bool energy = c_p.outputtype == otEnergy;
        float4* row = const_cast<float4*>(ps.rows()) + 3 * i;
        row[0] = make_float4(q.x, q.y, q.w, __fdividef(1.f, q.y));
        row[1] = make_float4(1.f - q.z * q.z, 1.f - q.z, 2.f * q.z, 1.f + q.z * q.z);
        row[2] = make_float4(__fdividef(1.f, 2.f * q.z), energy ? 1.f : __fdividef(1.f, q.x),
                             (!energy && q.x < K_EPS) ? 1.f : 0.f, 0.f);
    }
    for (unsigned int i = threadIdx.x; i < c_p.nangle; i += LB_BLOCK) {
        ps.tables()[i] = a.angleinvcdf[i];
    }
    __syncthreads();

    unsigned long long nfail = 0;
    Photon s;
    float cx = 0.f, cy = 0.f, cz = 0.f;    /* the voxel's centre */
    unsigned int m = 0;                    /* its byte: label and detector bit */
    unsigned int vt = 0, nsteps = 0, endflag = 0;
    /* the next step looks its voxel up even if it ends inside: a reflection leaves
       the voxel coordinates on the face's far side while the photon stays in the
       voxel it came from, and a point source's launch voxel comes without the
       detector bit */
    bool offgrid = false;
    s.f.x = 1.f;
    int st = (threadIdx.x & 31u) < a.lanes ? lb_claim(a, vt) : DONE;

    while (__any_sync(0xFFFFFFFFu, st != DONE)) {
        if (st == ENDED || st == FRESH) {
            bool go = true;
            if (st == ENDED && closephoton<DET != DET_NONE, false, false>(a, ps, S, s, endflag, vt)) {
                a.energy[vt] = make_float2(ps.cold()->esc, ps.cold()->launched);
                st = lb_claim(a, vt);
                go = st == FRESH;
            }
            if (go) {
                if (st == FRESH) {
                    vt_begin(a, ps, S, s, vt);
                }
                int r = 1;
                if (!(DET && st == FRESH && c_p.savedet == 3 && *(volatile unsigned int*)a.detcount >= c_p.maxdetphoton)) {
                    r = startphoton<false, DET != DET_NONE, false, false, false>(a, ps, S, s, vt, &nfail);
                }
                if (r) {
                    /* NO_LAUNCH: the reference's thread ends, without its energies if it launched nothing */
                    if (st == FRESH) {
                        atomicAdd(a.status + ST_FAILED_LAUNCH, 1u);
                    } else {
                        a.energy[vt] = make_float2(ps.cold()->esc, ps.cold()->launched);
                    }
                    st = lb_claim(a, vt);
                } else {
                    st = RUN;
                    nsteps = 0;
                    offgrid = true;
                    m = (s.mediaid & LB_LABEL) | ((s.mediaid & K_DET_MASK) >> 24);
                    cx = (float)s.fx + 0.5f;
                    cy = (float)s.fy + 0.5f;
                    cz = (float)s.fz + 0.5f;
                    s.f.x = lb_scatlen(s.t);
                }
            }
        }
        if (st == RUN) {
            const unsigned int label = m & LB_LABEL;
            if (s.f.x <= 0.f) {
                /* ---- scattering (mcx_core.cl:2446-2649) */
                s.f.x = lb_scatlen(s.t);
                float sphi, cphi;
                M::sincos(__fmul_rn(K_TWO_PI, __fsub_rn(rnd12(s.t), 1.f)), &sphi, &cphi);
                const float u = __fsub_rn(rnd12(s.t), 1.f);
                const float4 g = ps.row(label, 1);
                float ctheta = 2.f * u - 1.f;
                if (fabsf(g.z) > 2.f * K_EPS) {
                    const float t = __fmul_rn(g.x, rcp_approx(__fmaf_rn(g.z, u, g.y)));
                    ctheta = fmaxf(-1.f, fminf(1.f, __fmul_rn(__fmaf_rn(-t, t, g.w), ps.row(label, 2).x)));
                }
                const float stheta = M::sqrt(__fmaf_rn(-ctheta, ctheta, 1.f));
                if (DET == DET_SP || (DET == DET_ANY && SAVE_NSCAT(c_p.savedetflag))) {
                    float* q = &ps.slot(0, label);
                    *q = __uint_as_float(__float_as_uint(*q) + 1u);
                }
                if (DET == DET_ANY && SAVE_MOM(c_p.savedetflag)) {
                    ps.slot(SAVE_NSCAT(c_p.savedetflag) + SAVE_PPATH(c_p.savedetflag), label) += 1.f - ctheta;
                }
                rotate_rn(s.v, stheta, ctheta, sphi, cphi);
            }

            /* ---- move to the next voxel face or the end of the free path */
            const float4 A = ps.row(label, 0);
            const float4 h0 = c_h[0], h1 = c_h[1];
            const float sx = sign1(s.v.x), sy = sign1(s.v.y), sz = sign1(s.v.z);
            float hx = fabsf(__fmaf_rn(0.5f, sx, cx) - s.p.x);
            float hy = fabsf(__fmaf_rn(0.5f, sy, cy) - s.p.y);
            float hz = fabsf(__fmaf_rn(0.5f, sz, cz) - s.p.z);
            hx = fabsf((hx + K_EPS) * rcp_approx(s.v.x));
            hy = fabsf((hy + K_EPS) * rcp_approx(s.v.y));
            hz = fabsf((hz + K_EPS) * rcp_approx(s.v.z));
            float dist = fminf(fminf(hx, hy), hz);
            const bool px = dist == hx, py = !px & (dist == hy);
            const float slen = fminf(__fmul_rn(dist, A.y), s.f.x);
            dist = __fmul_rn(slen, A.w);
            s.pathlen = __fadd_rn(s.pathlen, dist);
            s.p.x = __fmaf_rn(dist, s.v.x, s.p.x);
            s.p.y = __fmaf_rn(dist, s.v.y, s.p.y);
            s.p.z = __fmaf_rn(dist, s.v.z, s.p.z);
            s.p.w = __fmul_rn(s.p.w, M::exp(__fmul_rn(-A.x, dist)));
            const bool cross = slen != s.f.x;
            s.f.x = __fsub_rn(s.f.x, slen);
            s.f.y = __fmaf_rn(__fmul_rn(dist, A.z), h0.w, s.f.y);
            if (DET == DET_P || DET == DET_SP || (DET == DET_ANY && SAVE_PPATH(c_p.savedetflag))) {
                float& q = ps.slot(DET == DET_P ? 0u : (DET == DET_SP ? 1u : SAVE_NSCAT(c_p.savedetflag)), label);
                q = __fadd_rn(q, dist);
            }
            const unsigned int mold = m, idxold = s.idx1d;
            nsteps++;
            bool event = (s.f.y > h1.x) | (fabsf(s.p.w) < h1.y) | (nsteps > K_STEP_CAP);
            const bool look = cross | offgrid;
            bool inside = true;
            if (look) {
                /* ---- new voxel (mcx_core.cl:2795-2811) */
                const float4 h2 = c_h[2], h3 = c_h[3];
                cx += (cross & px) ? sx : 0.f;
                cy += (cross & py) ? sy : 0.f;
                cz += (cross & !px & !py) ? sz : 0.f;
                offgrid = false;
                /* a float's bits order like the float from 0 up; a negative one's are above all */
                inside = (__float_as_uint(cx) < __float_as_uint(h0.x)) & (__float_as_uint(cy) < __float_as_uint(h0.y)) &
                         (__float_as_uint(cz) < __float_as_uint(h0.z));
                unsigned int idx = (unsigned int)((int)cz * __float_as_int(h2.w) + (int)cy * __float_as_int(h2.z) + (int)cx);
                idx = inside ? idx : idxold;
                m = __ldg(a.media8 + idx);
                /* ---- deposit on a voxel change (mcx_core.cl:2816-2929) */
                const bool left = (mold != 0u) & (!inside | (idx != idxold));
                const float4 C = ps.row(label, 2);
                const float weight = C.z > 0.f ? __fmul_rn(s.w0, s.pathlen) : __fmul_rn(__fsub_rn(s.w0, s.p.w), C.y);
                unsigned int key = idxold + (unsigned int)((int)floorf((s.f.y - h1.z) * h1.w)) * __float_as_uint(h3.x);
                /* a time of flight a rounding below the window's end folds into gate 0 */
                key = min(key, key - __float_as_uint(h3.y));
                if (left & (s.f.y >= h1.z) & (s.f.y < h1.x) & (fabsf(weight) > 0.f)) {
                    /* field_split and field_commit */
                    const float kf = rintf(__fmul_rn(weight, h2.x));
                    const float r = __fmaf_rn(-kf, h2.y, weight);
                    if (kf != 0.f) {
                        atomicAdd(a.fhi + key, (unsigned long long)__float2ll_rn(kf));
                    }
                    if (r != 0.f) {
                        atomicAdd(a.flo + key, r);
                    }
                }
                s.w0 = left ? s.p.w : s.w0;
                s.pathlen = left ? 0.f : s.pathlen;
                s.idx1d = idx;
                event = event | !inside | (((m ^ mold) & LB_LABEL) != 0u);
            }
            if (event) {
                bool stop = (s.f.y > c_p.twin1) | (nsteps > K_STEP_CAP), wrapped = false;
                unsigned int code = 0;
                s.fw = px ? 0 : (py ? 1 : 2);
                s.mediaid = look ? (m & LB_LABEL) : m;
                if (!inside) {
                    /* ---- at a face of the domain (mcx_core.cl:2958-3028) */
                    s.idx1d = (cx < 0.f || cy < 0.f || cz < 0.f) ? K_OUT_MIN : K_OUT_MAX;
                    code = c_p.bc[(s.idx1d == K_OUT_MAX) * 3 + s.fw];
                    code = ((code & 0xF) == bcUnknown) ? (c_p.doreflect ? bcReflect : bcAbsorb) : code;
                    s.mediaid = 0;
                    m = 0;
                    if (code == bcCyclic) {
                        if (s.fw == 0) {
                            s.p.x = nextafter_ref(rintf(((s.idx1d == K_OUT_MIN) ? c_p.maxidx.x : 0)), (s.v.x > 0.f) - (s.v.x < 0.f));
                            cx = floorf(s.p.x) + 0.5f;
                        } else if (s.fw == 1) {
                            s.p.y = nextafter_ref(rintf(((s.idx1d == K_OUT_MIN) ? c_p.maxidx.y : 0)), (s.v.y > 0.f) - (s.v.y < 0.f));
                            cy = floorf(s.p.y) + 0.5f;
                        } else {
                            s.p.z = nextafter_ref(rintf(((s.idx1d == K_OUT_MIN) ? c_p.maxidx.z : 0)), (s.v.z > 0.f) - (s.v.z < 0.f));
                            cz = floorf(s.p.z) + 0.5f;
                        }
                        wrapped = cx >= 0.f && cy >= 0.f && cz >= 0.f && cx < c_p.maxidx.x && cy < c_p.maxidx.y && cz < c_p.maxidx.z;
                        if (wrapped) {
                            s.idx1d = vox_index(ps, (int)cx, (int)cy, (int)cz);
                            m = __ldg(a.media8 + s.idx1d);
                        }
                    }
                    stop = !wrapped && (stop || code == bcAbsorb || code == bcCyclic || (code == bcReflect && A.z == ps.row(0, 0).z));
                } else if (!mold) {
                    /* a photon in the void stays there whatever it crosses into */
                    m &= LB_DET;
                    s.mediaid = 0;
                }
                endflag = lb_exitflag(s.idx1d, s.fw, mold);
                if (nsteps > K_STEP_CAP) {
                    atomicAdd(a.status + ST_GUARD, 1u);
                    endflag = 0;
                    stop = true;
                } else if (!stop && !wrapped && fabsf(s.p.w) < c_p.minenergy) {
                    /* ---- Russian roulette (mcx_core.cl:3031-3061) */
                    if (rnd(s.t) * K_ROULETTE <= 1.f) {
                        s.p.w *= K_ROULETTE;
                    } else {
                        stop = true;
                        endflag = (mold & LB_DET) << 24;
                    }
                }
                if (REFL && !stop && !wrapped && look && (((m ^ mold) & LB_LABEL) || code)) {
                    /* ---- Fresnel reflection / refraction (mcx_core.cl:3126-3278) */
                    const float n1 = A.z, n2 = ps.row(m & LB_LABEL, 0).z;
                    if ((((m & LB_LABEL) || code == bcUnknown) ? c_p.doreflect : (code == bcReflect || code == bcMirror)) &&
                        (code == bcMirror || n1 != n2)) {
                        float Rtotal = 1.f;
                        const float tmp0 = n1 * n1;
                        const float tmp1 = n2 * n2;
                        const float cphi = fabsf(vcomp(s.v, s.fw));
                        const float sphi = 1.f - cphi * cphi;
                        const float fz = 1.f - M::div(tmp0, tmp1) * sphi;
                        if (fz > 0.f && code != bcMirror) {
                            float ctheta = tmp0 * cphi * cphi + tmp1 * fz;
                            const float stheta = 2.f * n1 * n2 * cphi * M::sqrt(fz);
                            Rtotal = M::div(ctheta - stheta, ctheta + stheta);
                            ctheta = tmp1 * cphi * cphi + tmp0 * fz;
                            Rtotal = (Rtotal + M::div(ctheta - stheta, ctheta + stheta)) * 0.5f;
                        }
                        if (Rtotal < 1.f && code != bcMirror && rnd(s.t) > Rtotal) {
                            transmit<false>(s.v, n1, n2, s.fw);
                            stop = (m & LB_LABEL) == 0;
                        } else {
                            if (s.fw == 0) {
                                s.v.x = -s.v.x;
                                s.p.x = nextafter_ref(rintf(s.p.x), (int)((float)(s.v.x > 0.f) - 0.5f));
                                cx = rintf(s.p.x) + 0.5f;
                            } else if (s.fw == 1) {
                                s.v.y = -s.v.y;
                                s.p.y = nextafter_ref(rintf(s.p.y), (int)((float)(s.v.y > 0.f) - 0.5f));
                                cy = rintf(s.p.y) + 0.5f;
                            } else {
                                s.v.z = -s.v.z;
                                s.p.z = nextafter_ref(rintf(s.p.z), (int)((float)(s.v.z > 0.f) - 0.5f));
                                cz = rintf(s.p.z) + 0.5f;
                            }
                            s.idx1d = idxold;
                            m = __ldg(a.media8 + idxold);
                            offgrid = true;
                        }
                    }
                }
                if (stop) {
                    st = ENDED;
                }
            }
        }
    }
}

}  // namespace

cudaError_t label_upload(const mcxg_kparams* p, const float* det4, unsigned int ndet, cudaStream_t st) {
    cudaError_t e = cudaMemcpyToSymbolAsync(c_p, p, sizeof(*p), 0, cudaMemcpyHostToDevice, st);
    float h[16] = {p->maxidx.x, p->maxidx.y, p->maxidx.z, p->oneoverc0, p->twin1, p->minenergy, p->twin0, p->Rtstep,
                   p->fxscale, p->fxunit};
    const uint32_t hi[4] = {p->dimx, p->dimxy, p->nvox, p->fieldlen};
    memcpy(h + 10, hi, sizeof(hi));
    if (e == cudaSuccess) {
        e = cudaMemcpyToSymbolAsync(c_h, h, sizeof(h), 0, cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess && ndet) {
        e = cudaMemcpyToSymbolAsync(c_det, det4, sizeof(float) * 4 * ndet, 0, cudaMemcpyHostToDevice, st);
    }
    return e;
}

template <int DET>
static void* kdet(int flags) {
    return (flags & LF_REFL) ? (void*)mcx_transport_label<DET, true> : (void*)mcx_transport_label<DET, false>;
}

static void* select(int flags) {
    if (!(flags & LF_DET)) {
        return kdet<DET_NONE>(flags);
    }
    const int kinds = flags >> LF_KINDS & 0xF;     /* savedetflag's bits: 2 scatterings, 4 paths, 8 momentum */
    return kinds == 4 ? kdet<DET_P>(flags) : (kinds == 6 ? kdet<DET_SP>(flags) : kdet<DET_ANY>(flags));
}

cudaError_t label_launch(const KArgs& a, int flags, int grid, int block, size_t smem, cudaStream_t st) {
    void* f = select(flags);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            return e;
        }
    }
    void* args[] = {(void*)&a};
    return cudaLaunchKernel(f, dim3(grid), dim3(block), args, smem, st);
}

cudaError_t label_occupancy(int flags, int block, size_t smem, int* blocks_per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, select(flags), block, smem);
}

cudaError_t label_attributes(int flags, cudaFuncAttributes* attr) {
    return cudaFuncGetAttributes(attr, select(flags));
}

}  // namespace mcxg
