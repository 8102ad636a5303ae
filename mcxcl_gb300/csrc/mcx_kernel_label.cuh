/*
 * mcx_kernel_label.cuh -- the transport kernel of the usual configurations.
 *
 * Byte labels or float absorption, three dimensions, Henyey-Greenstein, one
 * source; deposits of flux, fluence or energy, their precision check, replays
 * and modulated sources -- each with all of that fixed at compile time.  The photons, their random numbers and every
 * rounding are those of mcx_transport (mcx_kernel.cuh), whose device
 * functions it shares; what differs is what a step costs.
 *
 * The kernel is bound by issue: a warp runs the scattering and the
 * voxel-crossing block in nearly every iteration, each with about half its
 * lanes, so the instructions of an iteration are what counts.  The cube +
 * sphere workload took 5,825 warp instructions a photon (counted by ncu) and
 * takes 3,780: no tests of what is fixed; nothing but deposits, label and
 * voxel index for the lanes that cross a face, and what is rare (faces of the
 * domain, label changes, time-outs, roulette) behind one test; conditions
 * combined without branches; voxel coordinates as floats; the parameters of a
 * step in four vector loads; a deposit scale per label instead of a choice of
 * output; what a replayed photon deposits looked up once, at its launch.
 * Kernel times before and after (one GB300; the small runs also by their
 * launch shape): cube, 1e4 photons 2.66 -> 1.23 ms, 1e6 8.95 -> 4.4 ms; cube +
 * sphere with detectors, 1e6 14.1 -> 7.1 ms, 2e7 113 -> 75 ms; head, 1e7 42.9 ->
 * 29 ms; modulated sphere, 1e6 17.2 -> 8.6 ms; replay of 9,000 photons 4.7 -> 1.75
 * ms; 1e6 photons on a 100^3 absorption map 13.3 -> 6.9 ms.
 */
#ifndef MCX_KERNEL_LABEL_CUH
#define MCX_KERNEL_LABEL_CUH

#include "mcx_kernel.cuh"
#include "mcx_launch.h"

namespace mcxg {
namespace {

constexpr int LB_BLOCK = kLabelBlock;     /* threads a block: shared-memory addresses are constants plus the lane's own */

/* The parameters a step reads, in the order in which it reads them and as
   vectors, so that four come with one load: {extents, 1/c0}, {window's end,
   roulette threshold, window's start, 1/gate}, {fixed-point scale and unit,
   dimx, dimxy}, {voxels, field length, 1 where energy is deposited, -}; extents
   and times are floats, the other sizes integers. */
#ifndef MCXG_BATCH_TU
__constant__ float4 c_h[4];
#endif

/* the same of one simulation, from its parameter block */
__device__ __forceinline__ float4 hot_of(const mcxg_kparams& k, int i) {
    return i == 0 ? make_float4(k.maxidx.x, k.maxidx.y, k.maxidx.z, k.oneoverc0)
           : i == 1 ? make_float4(k.twin1, k.minenergy, k.twin0, k.Rtstep)
           : i == 2 ? make_float4(k.fxscale, k.fxunit, __uint_as_float(k.dimx), __uint_as_float(k.dimxy))
           : make_float4(__uint_as_float(k.nvox), __uint_as_float(k.fieldlen), k.outputtype == otEnergy ? 1.f : 0.f, 0.f);
}

/* the three property rows of a medium {mua, mus, g, n} */
template <bool GEN>
__device__ __forceinline__ void lb_rows(float4* row, const float4& q, bool energy) {
    const float gg = __fmul_rn(q.z, q.z);
    row[0] = make_float4(q.x, q.y, q.w, __fdividef(1.f, q.y));
    row[1] = make_float4(GEN ? __fsub_rn(1.f, gg) : __fmaf_rn(-q.z, q.z, 1.f), 1.f - q.z, 2.f * q.z,
                         GEN ? __fadd_rn(1.f, gg) : __fmaf_rn(q.z, q.z, 1.f));
    row[2] = make_float4(__fdividef(1.f, 2.f * q.z), energy ? 1.f : __fdividef(1.f, q.x),
                         (!energy && q.x < K_EPS) ? 1.f : 0.f, 0.f);
}

/* the volume: a byte a voxel, label | detector bit << 7, or a word a voxel,
   absorption as a float whose sign is the detector bit */
enum { VOL_LABEL, VOL_MUA };

/* which partial data a run records: nothing, nothing but the detector, paths
   (the default 'dp'), paths and scattering counts ('dsp'), or whatever its
   flags say */
enum { DET_NONE, DET_ID, DET_P, DET_SP, DET_ANY };

/* what a lane is doing: a photon, waiting for its next one, for a claimed
   reference thread's first, or nothing more */
enum { RUNNING, ENDED, FRESH, DONE };

/* Parameter source.  Shared memory: three property rows a medium --
   {mua, mus, n, 1/mus}, {1 - g^2, 1 - g, 2g, 1 + g^2}, {1/(2g), deposit scale,
   1 where flux takes the path length itself, -} -- the launch-time states, the
   partial data, one slot for each label and kind (label 0's, a photon in a
   void voxel, which has no record, included: no update needs a test), and the
   launch angle table. */
#ifndef MCXG_BATCH_TU
template <int VOL, int DET>
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
    __device__ __forceinline__ float4 hot(int i) const { return c_h[i]; }
    template <bool GEN>
    __device__ __forceinline__ void stage(const KArgs& a) {
        for (unsigned int i = threadIdx.x; i < c_p.medianum; i += LB_BLOCK) {
            float4 q = a.gprop[i];
            if (VOL == VOL_MUA && i == 0 && c_p.medianum > 1) {
                /* scattering is medium 1's everywhere; a voxel without absorption has index 0's n */
                q.y = a.gprop[1].y;
                q.z = a.gprop[1].z;
            }
            lb_rows<GEN>(const_cast<float4*>(rows()) + 3 * i, q, c_p.outputtype == otEnergy);
        }
        for (unsigned int i = threadIdx.x; i < c_p.nangle; i += LB_BLOCK) {
            tables()[i] = a.angleinvcdf[i];
        }
    }
    /* the next reference thread that has photons: with fewer photons than
       threads, the threads from the photon count on have none */
    __device__ __forceinline__ int claim(const KArgs& a, unsigned int& vt) {
        vt = atomicAdd(a.vtcounter, 1u);
        return vt < c_p.nthread && (c_p.threadphoton || vt < (unsigned int)c_p.oddphoton) ? FRESH : DONE;
    }
    /* kinds of partial data */
    __device__ __forceinline__ unsigned int kinds() const {
        return DET == DET_ID ? 0u : DET == DET_P ? 1u : (DET == DET_SP ? 2u : SAVE_NSCAT(c_p.savedetflag) + SAVE_PPATH(c_p.savedetflag) + SAVE_MOM(c_p.savedetflag));
    }
    unsigned int tid;              /* opaque, so that it is kept and not read again at every use */
    __device__ __forceinline__ LabelPS() { asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid)); }
    __device__ __forceinline__ ColdState* cold() const { return (ColdState*)mcxg_smem + tid; }
    __device__ __forceinline__ const float4* rows() const { return mcxg_smem + LB_BLOCK * sizeof(ColdState) / sizeof(float4); }
    __device__ __forceinline__ const float4& row(unsigned int label, int k) const { return rows()[3 * label + k]; }
    __device__ __forceinline__ float4 prop(const Shared&, unsigned int i) const {
        const float4 q = row(VOL == VOL_MUA ? (unsigned int)(i != 0u) : i, 0);
        return make_float4(q.x, q.y, 0.f, q.z);
    }
    __device__ __forceinline__ float* slots() const { return (float*)(rows() + 3 * c_p.medianum); }
    __device__ __forceinline__ float& slot(unsigned int kind, unsigned int label) const {
        return slots()[(label * kinds() + kind) * LB_BLOCK + tid];
    }
    __device__ __forceinline__ void clear() const {
        if (DET != DET_NONE && DET != DET_ID) {
            const unsigned int n = kinds() * c_p.medianum;
            for (unsigned int i = 0; i < n; i++) {
                slots()[i * LB_BLOCK + tid] = 0.f;
            }
        }
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
#else
/* A batch: every simulation of the wave has its step parameters and property
   rows in shared memory, so that lanes of different simulations read theirs
   with one vector load as the lanes of one do; launches and rare events read
   the descriptor in constant memory.  A lane follows the simulation of the
   reference thread it claimed.  24 simulations of 2.3e6 photons: 97 ms with
   the parameters indexed in constant memory, where a warp whose lanes are in
   different simulations waits for each lane's load in turn, 11.7 ms so. */
template <int VOL, int DET>
struct LabelPS {
    static constexpr bool kBatch = true;
    static constexpr bool kXMedia = false;
    static constexpr bool kCommon = true;
    static constexpr int kHot = 5, kSim = kHot + 3 * MCXG_BATCH_MAXMEDIA;   /* float4s a simulation */
    unsigned int sid = 0;          /* the simulation of this wave */
    unsigned int lo;               /* remainder-plane offset: the batch's total field length */
    __device__ __forceinline__ const mcxg_kparams& p() const { return c_sims[sid].kp; }
    __device__ __forceinline__ const float4* det() const { return c_det; }   /* batches save no detectors */
    __device__ __forceinline__ const float4* srcx() const { return c_srcx; } /* nor use extra sources */
    __device__ __forceinline__ unsigned long long media_off() const { return c_sims[sid].media_off; }
    __device__ __forceinline__ unsigned int field_off() const { return (unsigned int)c_sims[sid].field_off; }
    __device__ __forceinline__ unsigned int lo_plane() const { return lo; }
    __device__ __forceinline__ unsigned long long vt_off() const { return c_sims[sid].vt_off; }
    __device__ __forceinline__ unsigned long long seed() const { return c_sims[sid].seed; }
    __device__ __forceinline__ ColdState* cold() const { return (ColdState*)mcxg_smem + threadIdx.x; }
    __device__ __forceinline__ const float4* sim() const {
        return mcxg_smem + LB_BLOCK * sizeof(ColdState) / sizeof(float4) + sid * kSim;
    }
    __device__ __forceinline__ float4 hot(int i) const { return sim()[i]; }
    __device__ __forceinline__ const float4& row(unsigned int label, int k) const { return sim()[kHot + 3 * label + k]; }
    __device__ __forceinline__ float4 prop(const Shared&, unsigned int i) const {
        const float4 q = row(i, 0);
        return make_float4(q.x, q.y, 0.f, q.z);
    }
    __device__ __forceinline__ float& slot(unsigned int, unsigned int) const { return *(float*)mcxg_smem; }
    __device__ __forceinline__ void clear() const {}
    __device__ __forceinline__ float& pp(unsigned int) const { return *(float*)mcxg_smem; }
    __device__ __forceinline__ float* tables() const { return (float*)mcxg_smem; }
    __device__ __forceinline__ float invcdf(unsigned int) const { return 0.f; }
    __device__ __forceinline__ float angle(unsigned int) const { return 0.f; }
    template <bool GEN>
    __device__ __forceinline__ void stage(const KArgs& a) {
        lo = a.lo;
        float4* base = const_cast<float4*>(sim());
        for (unsigned int i = threadIdx.x; i < a.nsim; i += LB_BLOCK) {
            const mcxg_simdesc& d = c_sims[i];
            float4* q = base + i * kSim;
            for (int k = 0; k < 4; k++) {
                q[k] = hot_of(d.kp, k);
            }
            q[4] = make_float4(__uint_as_float((unsigned int)d.media_off), __uint_as_float((unsigned int)(d.media_off >> 32)),
                               __uint_as_float((unsigned int)d.field_off), 0.f);
            for (int m = 0; m < MCXG_BATCH_MAXMEDIA; m++) {
                lb_rows<GEN>(q + kHot + 3 * m, f4(d.prop[m]), d.kp.outputtype == otEnergy);
            }
        }
    }
    /* As the other batch kernel's: the lane stays in its simulation until that
       one's counter has run out of threads with photons, then moves to the
       next open one */
    __device__ __forceinline__ int claim(const KArgs& a, unsigned int& vt) {
        for (;;) {
            if (sid < a.nsim) {
                const mcxg_kparams& k = c_sims[sid].kp;
                vt = atomicAdd(a.simctr + sid, 1u);
                if (vt < k.nthread && (k.threadphoton || vt < (unsigned int)k.oddphoton)) {
                    return FRESH;
                }
                atomicMax(a.vtcounter, sid + 1);
            }
            const unsigned int open = *(volatile unsigned int*)a.vtcounter;
            const unsigned int next = open > sid + 1 ? open : sid + 1;
            if (next >= a.nsim) {
                return DONE;
            }
            sid = next;
        }
    }
};
#endif

/* a voxel's value: its medium (label or absorption) and detector bit */
template <int VOL>
struct Voxel {
    static constexpr unsigned int kDet = VOL == VOL_MUA ? K_DET_MASK : 0x80u;
    static constexpr unsigned int kMedium = kDet - 1u;
    template <class PS>
    static __device__ __forceinline__ unsigned int load(const KArgs& a, const PS& ps, unsigned int idx) {
        if (PS::kBatch) {
            const float4 o = ps.hot(4);
            return __ldg(a.media8 + (((unsigned long long)__float_as_uint(o.y) << 32 | __float_as_uint(o.x)) + idx));
        }
        return VOL == VOL_MUA ? __ldg(a.media32 + idx) : (unsigned int)__ldg(a.media8 + idx);
    }
    /* the property row: the label, or whether there is any absorption */
    static __device__ __forceinline__ unsigned int row(unsigned int m) {
        return VOL == VOL_MUA ? (unsigned int)((m & kMedium) != 0u) : m & kMedium;
    }
    static __device__ __forceinline__ unsigned int detflag(unsigned int m) {
        return VOL == VOL_MUA ? m & K_DET_MASK : (m & kDet) << 24;
    }
};

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

/* The roundings of rotatevector and of the Henyey-Greenstein cosine as the
   compiler contracts them in mcx_transport, where a run of these
   configurations went before and some still go (other launch shapes,
   aggregated deposits): the photons stay the same to the bit.  GEN: as in the
   general instantiations, which float absorption and modulated sources took,
   rather than the common ones.  There the square of g
   and of the quotient are rounded by themselves, and the rotation's y starts
   from the other product. */
template <bool GEN>
__device__ __forceinline__ void rotate_rn(float4& v, float st, float ct, float sp, float cp) {
    const float t0 = __fmaf_rn(-v.z, v.z, 1.f);
    const float t1 = __fmul_rn(st, Mth<false>::rsqrt(t0));
    const float ix = __fmaf_rn(__fmul_rn(v.x, v.z), cp, -__fmul_rn(v.y, sp));
    const float yz = __fmul_rn(v.y, v.z);
    const float iy = GEN ? __fmaf_rn(yz, cp, __fmul_rn(v.x, sp)) : __fmaf_rn(v.x, sp, __fmul_rn(yz, cp));
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

/* the reference's detector flag of a photon that leaves (exit_detflag) */
template <int VOL>
__device__ __forceinline__ unsigned int lb_exitflag(const mcxg_kparams& c_p, unsigned int idx1d, int fw, unsigned int m) {
    return ((idx1d == K_OUT_MAX && c_p.bc[9 + fw]) || (idx1d == K_OUT_MIN && c_p.bc[6 + fw]))
           ? K_OUT_MIN : Voxel<VOL>::detflag(m);
}

/* field_add: the rounded product is a float integer, the remainder one exact fma */
__device__ __forceinline__ void lb_add(const KArgs& a, unsigned long long* hi, float* lo, unsigned int key, float w, float sc,
                                       float unit) {
    const float kf = rintf(__fmul_rn(w, sc));
    const float r = __fmaf_rn(-kf, unit, w);
    if (kf != 0.f) {
        atomicAdd(hi + key, (unsigned long long)__float2ll_rn(kf));
    }
    if (r != 0.f) {
        atomicAdd(lo + key, r);
    }
}

/* What a replayed photon deposits, fixed at its launch: the detected weight
   (x the time of flight where the output asks for it) and the offset of its
   gate and detector in the field (mcx_core.cl:2567-2604, 2845-2858).  The
   site outputs read the photon siteshift further on; one past the arrays
   deposits nothing, a gate or detector out of range counts in the status word
   at each deposit (kBad). */
struct Replayed {
    static constexpr unsigned int kBad = 0xFFFFFFFFu;
    float w, t;
    unsigned int off;
};

template <int KIND, class PS>
__device__ __forceinline__ Replayed replayed(const KArgs& a, const PS& ps, unsigned int vt, float launched) {
    Replayed q = {0.f, 1.f, 0u};
    const long long k = replay_index(ps, vt, (long long)(int)launched - 1 + (KIND == RUN_SITE ? (long long)c_p.siteshift : 0ll));
    if (k < 0 || k >= (long long)c_p.nreplay) {
        return q;
    }
    const float rt = __ldg(a.rtof + k);
    const int d = __ldg(a.rdetid + k) & 0xFFFF;
    int tshift = (int)(floorf((rt - c_p.twin0) * c_p.Rtstep)) + ((c_p.replaydet == -1) ? ((d - 1) * (int)c_p.maxgate) : 0);
    q.w = __ldg(a.rweight + k);
    if (KIND == RUN_JAC) {
        if (c_p.outputtype == otWLTOF) {
            q.t = rt;
        }
        if (tshift < 0 || (c_p.replaydet == -1 && (d < 1 || d > (int)c_p.detnum))) {
            q.off = Replayed::kBad;
        } else {
            q.off = (unsigned int)tshift * c_p.nvox;
        }
    } else {
        if (c_p.outputtype == otWPTOF) {
            q.w = __fmul_rn(rt, q.w);
        }
        tshift = ((int)c_p.maxgate - 1 < tshift) ? (int)c_p.maxgate - 1 : tshift;
        q.off = tshift < 0 ? Replayed::kBad : (unsigned int)tshift * c_p.nvox;
    }
    return q;
}

/* Every photon of a pencil beam without an angle table or focus, launched in
   a voxel with a medium, starts alike, with no random number: startphoton's
   result without its choice of sources (cube + sphere 2e7 photons 78.4 -> 75.7
   ms with the lane's index held in a register, head 1e7 31.2 -> 29.8; other
   sources' runs 2 % slower for the code between). */
__device__ __forceinline__ bool plainbeam(const mcxg_kparams& c_p) {
    return c_p.srctype == S_PENCIL && !c_p.nangle && c_p.srcdir.w == 0.f && !c_p.replay && c_p.maxvoidstep >= 2u &&
           (__float_as_uint(c_p.srcparam2.w) & K_MED_MASK) && fabsf(c_p.srcpos.w) > c_p.minenergy;
}

template <int DET, bool RF, class PS>
__device__ __forceinline__ void startbeam(const PS& ps, Photon& s) {
    const mcxg_kparams& c_p = ps.p();
    ps.clear();
    if (DET && c_p.issaveseed) {
        ps.cold()->ps0 = s.t.a;
        ps.cold()->ps1 = s.t.b;
    }
    s.p = f4(c_p.srcpos);
    s.v = f4(c_p.srcdir);
    s.f.x = 0.f;
    s.f.y = 0.f;
    s.idx1d = __float_as_uint(c_p.srcparam2.z);
    s.mediaid = __float_as_uint(c_p.srcparam2.w);
    s.fx = (int)(short)floorf(s.p.x);
    s.fy = (int)(short)floorf(s.p.y);
    s.fz = (int)(short)floorf(s.p.z);
    s.f.w += 1.f;
    ps.cold()->launched += s.p.w;
    ps.cold()->w0init = s.p.w;
    s.w0 = s.p.w;
    if (RF) {
        s.wre = s.w0re = s.p.w;
        s.wim = s.w0im = 0.f;
    }
}

template <int KIND, int VOL, int DET, bool REFL>
__global__ void __launch_bounds__(LB_BLOCK, KIND == RUN_RF || KIND == RUN_CHECK ? 3 : 4) mcx_transport_label(const KArgs a) {
    typedef Mth<false> M;
    typedef Voxel<VOL> V;
    constexpr bool GEN = VOL == VOL_MUA || KIND == RUN_RF;
    constexpr bool JAC = KIND == RUN_JAC, SITE = KIND == RUN_SITE, RF = KIND == RUN_RF;
    typedef LabelPS<VOL, DET> PS;
    PS ps;
    Shared S;
    S.bprop = S.brecip = a.gprop;
    ps.template stage<GEN>(a);
    __syncthreads();

    unsigned long long nfail = 0;
    Photon s;
    float cx = 0.f, cy = 0.f, cz = 0.f;    /* the voxel's centre */
    unsigned int m = 0;                    /* its value: medium and detector bit */
    unsigned int vt = 0, nsteps = 0, endflag = 0;
    /* the next step looks its voxel up even if it ends inside: a reflection leaves
       the voxel coordinates on the face's far side while the photon stays in the
       voxel it came from, and a point source's launch voxel comes without the
       detector bit */
    bool offgrid = false;
    s.f.x = 1.f;
    Replayed rp = {0.f, 1.f, 0u};
    int st = (threadIdx.x & 31u) < a.lanes ? ps.claim(a, vt) : DONE;

    while (__any_sync(0xFFFFFFFFu, st != DONE)) {
        if (st == ENDED || st == FRESH) {
            const mcxg_kparams& c_p = ps.p();
            bool go = true;
            if (st == ENDED && closephoton<DET != DET_NONE, false, false>(a, ps, S, s, endflag, vt)) {
                a.energy[ps.vt_off() + vt] = make_float2(ps.cold()->esc, ps.cold()->launched);
                st = ps.claim(a, vt);
                go = st == FRESH;
            }
            if (go) {
                if (st == FRESH) {
                    vt_begin(a, ps, S, s, vt);
                }
                int r = 1;
                if (!(DET && st == FRESH && c_p.savedet == 3 && *(volatile unsigned int*)a.detcount >= c_p.maxdetphoton)) {
                    if (plainbeam(ps.p())) {
                        startbeam<DET, RF>(ps, s);
                        r = 0;
                    } else {
                        r = startphoton<false, DET != DET_NONE, RF, false, false>(a, ps, S, s, vt, &nfail);
                    }
                }
                if (r) {
                    /* NO_LAUNCH: the reference's thread ends, without its energies if it launched nothing */
                    if (st == FRESH) {
                        atomicAdd(a.status + ST_FAILED_LAUNCH, 1u);
                    } else {
                        a.energy[ps.vt_off() + vt] = make_float2(ps.cold()->esc, ps.cold()->launched);
                    }
                    st = ps.claim(a, vt);
                } else {
                    st = RUNNING;
                    nsteps = 0;
                    offgrid = true;
                    /* a point source's voxel value comes from the host: bounded as the volume's are */
                    m = VOL == VOL_MUA ? s.mediaid : min(s.mediaid & V::kMedium, PS::kBatch ? MCXG_BATCH_MAXMEDIA - 1u : c_p.maxmedia) |
                        ((s.mediaid & K_DET_MASK) >> 24);
                    if (JAC || SITE) {
                        rp = replayed<KIND>(a, ps, vt, s.f.w);
                    }
                    cx = (float)s.fx + 0.5f;
                    cy = (float)s.fy + 0.5f;
                    cz = (float)s.fz + 0.5f;
                    s.f.x = lb_scatlen(s.t);
                }
            }
        }
        if (st == RUNNING) {
            const mcxg_kparams& c_p = ps.p();      /* in a batch, of the simulation just claimed */
            const unsigned int label = V::row(m);
            /* a float-absorption voxel is recorded under the label its bits spell, as ever: none but a denormal's */
            const bool recorded = VOL == VOL_LABEL || (m & V::kMedium) - 1u < c_p.maxmedia;
            if (s.f.x <= 0.f) {
                /* ---- scattering (mcx_core.cl:2446-2649) */
                s.f.x = lb_scatlen(s.t);
                float sphi, cphi;
                M::sincos(__fmul_rn(K_TWO_PI, __fsub_rn(rnd12(s.t), 1.f)), &sphi, &cphi);
                const float u = __fsub_rn(rnd12(s.t), 1.f);
                const float4 g = ps.row(label, 1);
                float ctheta;
                {
                    const float t = __fmul_rn(g.x, rcp_approx(__fmaf_rn(g.z, u, g.y)));
                    const float d = GEN ? __fsub_rn(g.w, __fmul_rn(t, t)) : __fmaf_rn(-t, t, g.w);
                    ctheta = fmaxf(-1.f, fminf(1.f, __fmul_rn(d, ps.row(label, 2).x)));
                    ctheta = fabsf(g.z) > 2.f * K_EPS ? ctheta : 2.f * u - 1.f;
                }
                const float stheta = M::sqrt(__fmaf_rn(-ctheta, ctheta, 1.f));
                if (DET == DET_SP || (DET == DET_ANY && SAVE_NSCAT(c_p.savedetflag) && recorded)) {
                    float* q = &ps.slot(0, VOL == VOL_MUA ? m & V::kMedium : label);
                    *q = __uint_as_float(__float_as_uint(*q) + 1u);
                }
                if (DET == DET_ANY && SAVE_MOM(c_p.savedetflag) && recorded) {
                    ps.slot(SAVE_NSCAT(c_p.savedetflag) + SAVE_PPATH(c_p.savedetflag), VOL == VOL_MUA ? m & V::kMedium : label) +=
                        1.f - ctheta;
                }
                rotate_rn<GEN>(s.v, stheta, ctheta, sphi, cphi);
                if (SITE) {
                    const unsigned int key = s.idx1d + rp.off;
                    if (rp.off != Replayed::kBad && key < c_p.fieldlen) {
                        lb_add(a, a.fhi, a.flo, key, c_p.outputtype == otDCS ? __fmul_rn(1.f - ctheta, rp.w) : rp.w, ps.hot(2).x, ps.hot(2).y);
                    } else {
                        atomicAdd(a.status + ST_GUARD, 1u);
                    }
                }
            }

            /* ---- move to the next voxel face or the end of the free path */
            float4 A = ps.row(label, 0);
            if (VOL == VOL_MUA) {
                A.x = fabsf(__uint_as_float(m));
            }
            const float4 h0 = ps.hot(0), h1 = ps.hot(1);
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
            if (RF) {
                /* w <- w exp(-(mua + i omega n / c0) ds) (mcx_core.cl:2750-2760) */
                const float att = M::exp(__fmul_rn(-A.x, dist));
                float rs, rc;
                M::sincos(c_p.omega * A.z * h0.w * dist, &rs, &rc);
                const float tre = att * (s.wre * rc + s.wim * rs);
                const float tim = att * (-s.wre * rs + s.wim * rc);
                s.wre = tre;
                s.wim = tim;
                s.p.w = M::sqrt(s.wre * s.wre + s.wim * s.wim);
            } else {
                s.p.w = __fmul_rn(s.p.w, M::exp(__fmul_rn(-A.x, dist)));
            }
            const bool cross = slen != s.f.x;
            s.f.x = __fsub_rn(s.f.x, slen);
            s.f.y = __fmaf_rn(__fmul_rn(dist, A.z), h0.w, s.f.y);
            if (DET == DET_P || DET == DET_SP || (DET == DET_ANY && SAVE_PPATH(c_p.savedetflag) && recorded)) {
                float& q = ps.slot(DET == DET_P ? 0u : (DET == DET_SP ? 1u : SAVE_NSCAT(c_p.savedetflag)),
                                   VOL == VOL_MUA ? m & V::kMedium : label);
                q = __fadd_rn(q, dist);
            }
            const unsigned int mold = m, idxold = s.idx1d;
            nsteps++;
            const bool over = s.f.y > h1.x;
            bool event = over | (fabsf(s.p.w) < h1.y) | (nsteps > K_STEP_CAP);
            const bool look = cross | offgrid;
            bool inside = true;
            if (look) {
                /* ---- new voxel (mcx_core.cl:2795-2811) */
                const float4 h2 = ps.hot(2), h3 = ps.hot(3);
                if (cross & px) {
                    cx += sx;
                }
                if (cross & py) {
                    cy += sy;
                }
                if (cross & !px & !py) {
                    cz += sz;
                }
                offgrid = false;
                /* a float's bits order like the float from 0 up; a negative one's are above all */
                inside = (__float_as_uint(cx) < __float_as_uint(h0.x)) & (__float_as_uint(cy) < __float_as_uint(h0.y)) &
                         (__float_as_uint(cz) < __float_as_uint(h0.z));
                unsigned int idx = (unsigned int)((int)cz * __float_as_int(h2.w) + (int)cy * __float_as_int(h2.z) + (int)cx);
                idx = inside ? idx : idxold;
                m = V::load(a, ps, idx);
                /* ---- deposit on a voxel change (mcx_core.cl:2816-2929) */
                const bool left = (mold != 0u) & (!inside | (idx != idxold));
                const bool inwin = (s.f.y >= h1.z) & (s.f.y < h1.x);
                if (JAC) {
                    const float weight = __fmul_rn(__fmul_rn(rp.w, s.pathlen), rp.t);
                    if (left & inwin & (rp.off == Replayed::kBad)) {
                        atomicAdd(a.status + ST_GUARD, 1u);
                    } else if (left & inwin & (fabsf(weight) > 0.f)) {
                        unsigned int key = idxold + rp.off;
                        key = min(key, key - __float_as_uint(h3.y));
                        lb_add(a, a.fhi, a.flo, key, weight, h2.x, h2.y);
                    }
                } else if (!SITE) {
                    unsigned int key = idxold + (unsigned int)((int)floorf((s.f.y - h1.z) * h1.w)) * __float_as_uint(h3.x);
                    /* a time of flight a rounding below the window's end folds into gate 0 */
                    key = min(key, key - __float_as_uint(h3.y));
                    float weight;
                    if (RF) {
                        /* (w0 - w) / (mua + i omega n / c0) (mcx_core.cl:2833-2840) */
                        const float dre = s.w0re - s.wre, dim = s.w0im - s.wim;
                        const float aim = c_p.omega * A.z * h0.w;
                        const float am2 = A.x * A.x + aim * aim;
                        weight = (am2 < K_EPS) ? (s.w0re * s.pathlen) : M::div(dre * A.x + dim * aim, am2);
                        const float weight_im = (am2 < K_EPS) ? (s.w0im * s.pathlen) : M::div(dim * A.x - dre * aim, am2);
                        if (left & inwin & (fabsf(weight) > 0.f)) {
                            lb_add(a, a.fhi + c_p.fieldlen, a.flo + c_p.fieldlen, key, weight_im, h2.x, h2.y);
                        }
                    } else if (VOL == VOL_MUA) {
                        const float loss = __fsub_rn(s.w0, s.p.w);
                        weight = A.x < K_EPS ? __fmul_rn(s.w0, s.pathlen) : __fmul_rn(loss, rcp_approx(A.x));
                        weight = h3.z != 0.f ? loss : weight;
                    } else {
                        const float4 C = ps.row(label, 2);
                        weight = C.z > 0.f ? __fmul_rn(s.w0, s.pathlen) : __fmul_rn(__fsub_rn(s.w0, s.p.w), C.y);
                    }
                    if (left & (s.f.y >= h1.z) & (s.f.y < h1.x) & (fabsf(weight) > 0.f)) {
                        /* field_split and field_commit: the rounded product is a float
                           integer, the remainder one exact fma */
                        const float kf = rintf(__fmul_rn(weight, h2.x));
                        const float r = __fmaf_rn(-kf, h2.y, weight);
                        if (PS::kBatch) {
                            key += __float_as_uint(ps.hot(4).z);
                        }
                        atomicAdd(a.fhi + key, (unsigned long long)__float2ll_rn(kf));
                        if (r != 0.f) {
                            atomicAdd(a.flo + key, r);
                        }
                        if (KIND == RUN_CHECK) {
                            acc_verify(a, ps.lo_plane(), key, weight);
                        }
                    }
                }
                if (RF) {
                    s.w0re = left ? s.wre : s.w0re;
                    s.w0im = left ? s.wim : s.w0im;
                }
                s.w0 = left ? s.p.w : s.w0;
                s.pathlen = left ? 0.f : s.pathlen;
                s.idx1d = idx;
                event = event | !inside | (VOL == VOL_MUA ? V::row(m) != label : ((m ^ mold) & V::kMedium) != 0u);
            }
            if (event) {
                bool stop = over | (nsteps > K_STEP_CAP), wrapped = false;
                unsigned int code = 0;
                s.fw = px ? 0 : (py ? 1 : 2);
                s.mediaid = look ? (m & V::kMedium) : m;
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
                            m = V::load(a, ps, s.idx1d);
                        }
                    }
                    stop = !wrapped && (stop || code == bcAbsorb || code == bcCyclic || (code == bcReflect && A.z == ps.row(0, 0).z));
                } else if (!mold) {
                    /* a photon in the void stays there whatever it crosses into */
                    m &= V::kDet;
                    s.mediaid = 0;
                }
                endflag = lb_exitflag<VOL>(c_p, s.idx1d, s.fw, mold);
                if (nsteps > K_STEP_CAP) {
                    atomicAdd(a.status + ST_GUARD, 1u);
                    endflag = 0;
                    stop = true;
                } else if (!stop && !wrapped && fabsf(s.p.w) < c_p.minenergy) {
                    /* ---- Russian roulette (mcx_core.cl:3031-3061) */
                    if (rnd(s.t) * K_ROULETTE <= 1.f) {
                        s.p.w *= K_ROULETTE;
                        if (RF) {
                            s.wre *= K_ROULETTE;
                            s.wim *= K_ROULETTE;
                            s.w0re *= K_ROULETTE;
                            s.w0im *= K_ROULETTE;
                        }
                    } else {
                        stop = true;
                        endflag = V::detflag(mold);
                    }
                }
                if (REFL && !stop && !wrapped && look && (V::row(m) != label || code)) {
                    /* ---- Fresnel reflection / refraction (mcx_core.cl:3126-3278) */
                    const float n1 = A.z, n2 = ps.row(V::row(m), 0).z;
                    if ((((m & V::kMedium) || code == bcUnknown) ? c_p.doreflect : (code == bcReflect || code == bcMirror)) &&
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
                            stop = (m & V::kMedium) == 0;
                        } else {
                            /* nextafter_ref's step is 0 here (its direction of +-0.5 becomes the
                               integer 0): the coordinate is the face's */
                            if (s.fw == 0) {
                                s.v.x = -s.v.x;
                                s.p.x = __fadd_rn(rintf(s.p.x), 0.f);
                                cx = s.p.x + 0.5f;
                            } else if (s.fw == 1) {
                                s.v.y = -s.v.y;
                                s.p.y = __fadd_rn(rintf(s.p.y), 0.f);
                                cy = s.p.y + 0.5f;
                            } else {
                                s.v.z = -s.v.z;
                                s.p.z = __fadd_rn(rintf(s.p.z), 0.f);
                                cz = s.p.z + 0.5f;
                            }
                            s.idx1d = idxold;
                            m = V::load(a, ps, idxold);
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
}  // namespace mcxg

#endif
