// sfp_step.cuh -- the fused particle step: every species of every instance by
// one step in three launches (massive, photon, appends), or several steps in
// one launch where the population is small (sfp_steps_body).
//
// Compiled by NVRTC together with a generated field program that defines
//     SFP_DEVICE_INLINE void sfp_field_program(double x, double y, double z,
//                                              double t, const double* P, double F[6]);
// so the field expression is inlined into the push.
//
// Semantics follow simulation.py:102-144 exactly:
//   1. fields at t for pushed species (particles.py:299-323),
//   2. chi + pair events for photon species (QED at t),
//   3. chi + photon events + hard-photon filter for e+- species,
//   4. photons appended (e- species first, in buffer order), recoil,
//   5. pairs appended, converted photons pruned,
//   6. every pushed particle -- children included -- pushed from t to t+dt:
//      half position, fields at t+dt/2, Boris / Boris-TBMT (+LL/CLL), half position.
// A call's first step is prepared by a one-block kernel (sfp_book_kernel); a
// step is:
//   massive -- 3; a particle with an event is marked and left as it was at t
//              (its delta stored), every other one takes 6;
//   photon  -- 2; a converted photon is marked (its delta stored), every
//              other one takes 6.  Calls of several steps with many photons
//              visit only the photons that could convert, from a store of
//              them (sfp_hot_*);
//   step end, in the last block of the photon launch -- the children's slots:
//              per-tile event counts scanned in the reference's order; the
//              next step planned (sfp_step_end);
//   appends -- 4 (child from the parent's state at t, then the parent's
//              recoil and 6) and 5 (children pushed, 6), at those slots.
// The massive and photon kernels touch disjoint memory: each writes only
// below the start-of-step counts of its own group's buffers.  Appends are
// ordered: a child gets the slot that the reference's find_event_index +
// create_* would give it, so Philox streams keyed by slot are reproducible.
// Only the one-launch kernel's blocks wait on one another, at grid barriers of
// a cooperative launch, each wait with a time limit (sfp_grid_barrier).
#pragma once
#include "sfp_device.cuh"
#include "sfp_device32.cuh"
#include "sfp_mlp.cuh"
#include "sfp_run.cuh"

// threads per block of the group kernels (8 warps, each on its own tiles)
#ifndef SFP_TILE
#define SFP_TILE 256
#endif
// tiles per super-tile of the event scan
#define SFP_SUPER_TILE 64
// pruned-flag value of a particle whose event of this step awaits its children
#define SFP_MARK 2

namespace sfp {

SFP_DEVICE_INLINE unsigned int u4_get(const uint4& v, int c) {
    return c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : v.w;
}
SFP_DEVICE_INLINE uint4 u4_one(int c, unsigned int n) {
    uint4 v{0u, 0u, 0u, 0u};
    if (c == 0) v.x = n;
    else if (c == 1) v.y = n;
    else if (c == 2) v.z = n;
    else v.w = n;
    return v;
}
SFP_DEVICE_INLINE uint4 u4_add(uint4 a, uint4 b) { return uint4{a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w}; }

// Asynchronous 16-byte global -> shared copies (cp.async, one per thread,
// L2 only); `src_bytes` < 16 zero-fills the rest and reads only that many.
// Issue and commit carry no "memory" clobber, so values the compiler holds in
// registers survive them; the destination's earlier readers are ordered by
// the caller's __syncwarp() before the issue (volatile asm is not moved across
// it), and the data is read only after cp_async_wait, which is a clobber.
SFP_DEVICE_INLINE void cp_async16(void* smem_dst, const void* gsrc, unsigned int src_bytes) {
    const unsigned int d = (unsigned int)__cvta_generic_to_shared(smem_dst);
    const unsigned long long g = (unsigned long long)__cvta_generic_to_global(gsrc);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(g), "r"(src_bytes));
}
SFP_DEVICE_INLINE void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
SFP_DEVICE_INLINE void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// inclusive / exclusive warp sums
SFP_DEVICE_INLINE unsigned int warp_incl_scan(unsigned int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    return v;
}
SFP_DEVICE_INLINE unsigned int warp_sum(unsigned int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// bit b set where byte b of the 16 bytes v equals SFP_MARK
SFP_DEVICE_INLINE unsigned int marks16(uint4 v) {
    const unsigned int k = SFP_MARK * 0x01010101u;
    const unsigned int w[4] = {__vcmpeq4(v.x, k), __vcmpeq4(v.y, k), __vcmpeq4(v.z, k), __vcmpeq4(v.w, k)};
    unsigned int m = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        m |= (((w[q] >> 7) & 1u) | ((w[q] >> 14) & 2u) | ((w[q] >> 21) & 4u) | ((w[q] >> 28) & 8u)) << (4 * q);
    return m;
}

// Push of one massive particle from t to t+dt (simulation.py:128-137 with
// particles.py:244-296 / 575-604).  x, u (and s) in/out.
SFP_DEVICE_INLINE void push_massive(double& x, double& y, double& z, double& ux, double& uy, double& uz, double& sx,
                                    double& sy, double& sz, const sfp_segment& S, const double* __restrict__ P,
                                    double t, double dt) {
    double ig = inv_gamma_massive(ux, uy, uz);
    push_position(x, y, z, ux, uy, uz, ig, 0.5 * dt);
    double F[6];
    sfp_field_program(x, y, z, t + 0.5 * dt, P, F);
    if (S.spin)
        ig = boris_tbmt(ux, uy, uz, sx, sy, sz, F, S.q, S.ae, dt);
    else
        ig = boris(ux, uy, uz, F, S.q, dt);
    if (S.rr == SFP_RR_LL || (S.rr == SFP_RR_CLL && !S.spin)) {
        const double chi = chi_of(F, ux, uy, uz, ig);
        ig = ll_push(ux, uy, uz, ig, chi, dt, S.rr == SFP_RR_CLL);
    }
    push_position(x, y, z, ux, uy, uz, ig, 0.5 * dt);
}

SFP_DEVICE_INLINE void push_photon(double& x, double& y, double& z, double ux, double uy, double uz, double dt) {
    const double ig = inv_gamma_photon(ux, uy, uz);
    push_position(x, y, z, ux, uy, uz, ig, 0.5 * dt);
    push_position(x, y, z, ux, uy, uz, ig, 0.5 * dt);
}

// float32 form of push_massive: float32 increments, float64 accumulation.
// The float32 push's per-(segment, step) constants, formed once per tile
// rather than once per particle (the same expressions, so the same values)
struct sfp_pc32 {
    double th;  // t + dt/2, the time of the push's field
    float hc;   // c dt / 2
    float eps;  // q dt / (2 m c)
    float bq;   // q dt / (2 m)
    float ll;   // the LL / CLL prefactor
};

SFP_DEVICE_INLINE sfp_pc32 push_consts32(const sfp_segment& S, double t, double dt) {
    sfp_pc32 K;
    K.th = t + 0.5 * dt;
    K.hc = (float)(0.5 * kC * dt);
    K.eps = (float)((S.q * dt) / ((2.0 * kMe) * kC));
    K.bq = (float)((S.q * dt) / (2.0 * kMe));
    K.ll = (float)ll_factor(dt);
    return K;
}

// The float32 push's sums of products have their roundings spelled out: which
// product of a sum a compiler fuses depends on the code around it, so the same
// source rounded differently in the group kernels, the appends kernel and the
// one-launch kernel, and one float32 ulp of a momentum is enough to turn a
// later event.  Now every kernel rounds alike (a b - c d: the second product is
// rounded first).
SFP_DEVICE_INLINE float diff_of_products(float a, float b, float c, float d) { return __fmaf_rn(a, b, -__fmul_rn(c, d)); }
SFP_DEVICE_INLINE float gamma_push(double ux, double uy, double uz) {
    const float fx = sfp32::d2f(ux), fy = sfp32::d2f(uy), fz = sfp32::d2f(uz);
    const float u2 = __fmaf_rn(fz, fz, __fmaf_rn(fx, fx, __fmul_rn(fy, fy)));
    if (u2 < (float)(sfp32::kGammaSplit * sfp32::kGammaSplit)) return sqrtf(1.0f + u2);
    return sfp32::d2f(sqrt(((1.0 + ux * ux) + uy * uy) + uz * uz));
}

// CHILD: a push in the step of an event (emitters and new pairs, appends kernel)
template <bool CHILD>
SFP_DEVICE_INLINE void push_massive32(double& x, double& y, double& z, double& ux, double& uy, double& uz,
                                      double& sx, double& sy, double& sz, const sfp_segment& S,
                                      const double* __restrict__ P, const sfp_pc32& K) {
    const float hc = K.hc;
    float g = gamma_push(ux, uy, uz);
    float fx = sfp32::d2f(ux), fy = sfp32::d2f(uy), fz = sfp32::d2f(uz);
    float a = __fdividef(hc, g);
    x += (double)(a * fx);
    y += (double)(a * fy);
    z += (double)(a * fz);
    float F[6];
    sfp_field_program32(x, y, z, K.th, P, F);
    const float eps = K.eps;
    const float bq = K.bq;
    const float ex = eps * F[0], ey = eps * F[1], ez = eps * F[2];
    const float umx = CHILD ? __fadd_rn(fx, ex) : __fmaf_rn(eps, F[0], fx);
    const float umy = CHILD ? __fadd_rn(fy, ey) : __fmaf_rn(eps, F[1], fy);
    const float umz = CHILD ? __fadd_rn(fz, ez) : __fmaf_rn(eps, F[2], fz);
    float gm;
    if (g < (float)sfp32::kGammaSplit) {
        gm = sqrtf(1.0f + umx * umx + umy * umy + umz * umz);
    } else {
        const double dx = ux + (double)ex, dy = uy + (double)ey, dz = uz + (double)ez;
        gm = sfp32::d2f(sqrt(((1.0 + dx * dx) + dy * dy) + dz * dz));
    }
    const float igm = __fdividef(1.0f, gm);
    if (S.spin) {  // inline.py:39-70: spin rotation with B_eff(u-), as an increment
        const float ae = sfp32::d2f(S.ae);
        const float uB = umx * F[3] + umy * F[4] + umz * F[5];
        const float a1 = ae + igm, a2 = __fdividef(ae * gm, gm + 1.0f), a3 = ae + __fdividef(1.0f, gm + 1.0f);
        const float bex = a1 * F[3] - a2 * uB * umx - a3 * (umy * F[2] - umz * F[1]);
        const float bey = a1 * F[4] - a2 * uB * umy - a3 * (umz * F[0] - umx * F[2]);
        const float bez = a1 * F[5] - a2 * uB * umz - a3 * (umx * F[1] - umy * F[0]);
        const float Tx = bq * bex, Ty = bq * bey, Tz = bq * bez;
        const float f2 = __fdividef(2.0f, 1.0f + Tx * Tx + Ty * Ty + Tz * Tz);
        const float s0x = sfp32::d2f(sx), s0y = sfp32::d2f(sy), s0z = sfp32::d2f(sz);
        const float spx = s0x + (s0y * Tz - s0z * Ty), spy = s0y + (s0z * Tx - s0x * Tz), spz = s0z + (s0x * Ty - s0y * Tx);
        sx += (double)(f2 * (spy * Tz - spz * Ty));
        sy += (double)(f2 * (spz * Tx - spx * Tz));
        sz += (double)(f2 * (spx * Ty - spy * Tx));
    }
    // Boris (inline.py:4-36) as u += 2 eps E + u' x S
    const float Tx = bq * F[3] * igm, Ty = bq * F[4] * igm, Tz = bq * F[5] * igm;
    const float upx = umx + diff_of_products(umy, Tz, umz, Ty), upy = umy + diff_of_products(umz, Tx, umx, Tz),
                upz = umz + diff_of_products(umx, Ty, umy, Tx);
    const float f2 = __fdividef(2.0f, 1.0f + Tx * Tx + Ty * Ty + Tz * Tz);
    ux += (double)__fadd_rn(2.0f * ex, f2 * diff_of_products(upy, Tz, upz, Ty));
    uy += (double)__fadd_rn(2.0f * ey, f2 * diff_of_products(upz, Tx, upx, Tz));
    uz += (double)__fadd_rn(2.0f * ez, f2 * diff_of_products(upx, Ty, upy, Tx));
    g = gamma_push(ux, uy, uz);
    if (S.rr == SFP_RR_LL || (S.rr == SFP_RR_CLL && !S.spin)) {  // inline.py:104-123
        fx = sfp32::d2f(ux); fy = sfp32::d2f(uy); fz = sfp32::d2f(uz);
        const float chi = sfp32::chi_of(F, fx, fy, fz, g);
        float factor = K.ll;
        if (S.rr == SFP_RR_CLL) {
            const float q = 1.0f + 4.8f * (1.0f + chi) * __logf(1.0f + 1.7f * chi) + 2.44f * chi * chi;
            factor *= exp2f(-0.66666667f * __log2f(q));
        }
        const float c = __fdividef(factor * chi * chi, g);
        ux += (double)(c * fx);
        uy += (double)(c * fy);
        uz += (double)(c * fz);
        g = sfp32::gamma_of(ux, uy, uz, false);
    }
    a = __fdividef(hc, g);
    x += (double)(a * sfp32::d2f(ux));
    y += (double)(a * sfp32::d2f(uy));
    z += (double)(a * sfp32::d2f(uz));
}

SFP_DEVICE_INLINE void push_photon32(double& x, double& y, double& z, double ux, double uy, double uz, double dt) {
    const float fx = sfp32::d2f(ux), fy = sfp32::d2f(uy), fz = sfp32::d2f(uz);
    const float a = sfp32::d2f(kC * dt) * rsqrtf(fx * fx + fy * fy + fz * fz);
    x += (double)(a * fx);
    y += (double)(a * fy);
    z += (double)(a * fz);
}

// n steps of the photon push at once (n may be negative): a photon's
// momentum does not change while it flies, so n pushes add n times the same
// displacement.  float64: each push adds ((c dt/2) / |u|) u twice (cpu.py:
// 5-19 with dt/2, push_photon); float32: (c dt / |u|) u as one float32
// increment (push_photon32).  Equal to n successive pushes up to the
// rounding of the float64 sum.
template <int FORM>
SFP_DEVICE_INLINE void photon_shift(double& x, double& y, double& z, double ux, double uy, double uz, double dt,
                                    double n) {
    if (FORM == SFP_FORM_FP64) {
        const double k = ((kC * (0.5 * dt)) * inv_gamma_photon(ux, uy, uz)) * (2.0 * n);
        x += k * ux;
        y += k * uy;
        z += k * uz;
    } else {
        const float fx = sfp32::d2f(ux), fy = sfp32::d2f(uy), fz = sfp32::d2f(uz);
        const float a = sfp32::d2f(kC * dt) * rsqrtf(fx * fx + fy * fy + fz * fz);
        x += n * (double)(a * fx);
        y += n * (double)(a * fy);
        z += n * (double)(a * fz);
    }
}

}  // namespace sfp

#if defined(SFP_WANT_STEP)

// ---------------------------------------------------------------------------
// Field parameters.  A module built for runs of one instance (a Simulation)
// defines SFP_CONST_FIELD_N, the length of its field's parameter block, and
// reads the block from this module's constant bank: the field program's
// reads are at compile-time offsets, so they become constant operands of
// the arithmetic instead of loads.  The host copies the run's block into
// sfp_cfield on the run's stream before each launch sequence (sfp_capi.cu,
// runs sharing a module are ordered).  Modules for several instances read
// each instance's block from global memory.
// ---------------------------------------------------------------------------
#if defined(SFP_CONST_FIELD_N)
// (a variable at global scope: its name is not mangled)
__constant__ __align__(16) double sfp_cfield[SFP_CONST_FIELD_N];
#endif

SFP_DEVICE_INLINE const double* sfp_field_params(const sfp_instance& I) {
#if defined(SFP_CONST_FIELD_N)
    (void)I;
    return sfp_cfield;
#else
    return I.field_params;
#endif
}

// The step's rejection-sampling draws: Philox-4x32-10 keyed by the instance
// seed (sfp::uniform2 / sfp32::uniform2f).  A one-instance module takes the
// ten rounds' keys (the seed's key schedule, k0 and k1 per round) from its
// constant bank, copied by the host with the field parameters, instead of
// forming them with two additions per round: the same numbers.
#if defined(SFP_CONST_FIELD_N)
__constant__ unsigned int sfp_ckeys[20];
#endif

SFP_DEVICE_INLINE sfp::U4 sfp_step_philox(sfp::U4 c, unsigned long long seed) {
#if defined(SFP_CONST_FIELD_N)
    (void)seed;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const unsigned int lo0 = 0xD2511F53u * c.x;
        const unsigned int hi0 = __umulhi(0xD2511F53u, c.x);
        const unsigned int lo1 = 0xCD9E8D57u * c.z;
        const unsigned int hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = sfp::U4{hi1 ^ c.y ^ sfp_ckeys[2 * r], lo1, hi0 ^ c.w ^ sfp_ckeys[2 * r + 1], lo0};
    }
    return c;
#else
    return sfp::philox4x32_10(c, (unsigned int)seed, (unsigned int)(seed >> 32));
#endif
}

SFP_DEVICE_INLINE void sfp_step_uniform2(unsigned long long seed, unsigned int stream, unsigned int step,
                                         unsigned int purpose, long long slot, double& r1, double& r2) {
    const sfp::U4 o = sfp_step_philox(sfp::philox_counter(stream, step, purpose, slot), seed);
    r1 = sfp::u01(o.x, o.y);
    r2 = sfp::u01(o.z, o.w);
}

SFP_DEVICE_INLINE void sfp_step_uniform2f(unsigned long long seed, unsigned int stream, unsigned int step,
                                          unsigned int purpose, long long slot, float& r1, float& r2) {
    sfp32::uniform2f_of(sfp_step_philox(sfp::philox_counter(stream, step, purpose, slot), seed), r1, r2);
}

// ---------------------------------------------------------------------------
// QED tables staged in shared memory (float64, or float32 copies for FP32)
// ---------------------------------------------------------------------------
struct sfp_qed_smem {
    const double* iAt;
    const double* dAt;
    const float* iAf;
    const float* dAf;
    const double* od_ph;
    const double* od_pa;
    int zN;
    double zmax;
    float inv_dzf;
    float base_maxf;
    double chi_pair_min;  // below: no pair event is possible (z_min > z_max)
    double od_chi_min_ph, od_chi_min_pa;  // optical depth: 10^log_chi_min of each table
    const float* od_phf;  // float32 form, optical depth: the total-rate tables as float32
    const float* od_paf;
};

template <int FORM, int QED>
__device__ __forceinline__ sfp_qed_smem sfp_stage_tables(const sfp_run_dev* __restrict__ R, double* s_tab) {
    sfp_qed_smem T;
    T.iAt = T.dAt = s_tab;
    T.iAf = T.dAf = reinterpret_cast<const float*>(s_tab);
    T.od_ph = T.od_pa = s_tab;
    T.od_phf = T.od_paf = reinterpret_cast<const float*>(s_tab);
    T.zN = 0;
    T.zmax = 0.0;
    if (QED == SFP_QED_REJECTION) {
        T.zN = R->rs.z_N;
        T.zmax = R->rs.z_max;
        if (FORM == SFP_FORM_FP64) {
            for (int i = threadIdx.x; i < T.zN; i += blockDim.x) {
                s_tab[i] = R->rs.int_Ai[i];
                s_tab[T.zN + i] = R->rs.Aip[i];
            }
            T.dAt = s_tab + T.zN;
        } else {
            float* f = reinterpret_cast<float*>(s_tab);
            for (int i = threadIdx.x; i < T.zN; i += blockDim.x) {
                f[i] = (float)R->rs.int_Ai[i];
                f[T.zN + i] = (float)R->rs.Aip[i];
            }
            T.dAf = f + T.zN;
        }
    } else {
        const int n1 = R->od_photon.chi_N, n2 = R->od_pair.chi_N;
        if (FORM == SFP_FORM_FP64) {
            for (int i = threadIdx.x; i < n1; i += blockDim.x) s_tab[i] = R->od_photon.rate_total[i];
            for (int i = threadIdx.x; i < n2; i += blockDim.x) s_tab[n1 + i] = R->od_pair.rate_total[i];
            T.od_pa = s_tab + n1;
        } else {
            float* f = reinterpret_cast<float*>(s_tab);
            for (int i = threadIdx.x; i < n1; i += blockDim.x) f[i] = (float)R->od_photon.rate_total[i];
            for (int i = threadIdx.x; i < n2; i += blockDim.x) f[n1 + i] = (float)R->od_pair.rate_total[i];
            T.od_paf = f + n1;
        }
    }
    T.inv_dzf = (float)((double)(T.zN - 1) / T.zmax);
    T.base_maxf = (float)(T.zmax * sqrt(T.zmax));
    // pair creation needs z_min = (4/chi)^(2/3) <= z_max: exact cut with margin
    T.chi_pair_min = QED == SFP_QED_REJECTION ? 4.0 / (T.zmax * sqrt(T.zmax)) * (1.0 - 1e-6) : 0.0;
    T.od_chi_min_ph = QED == SFP_QED_OPTICAL_DEPTH ? pow(10.0, R->od_photon.log_chi_min) : 0.0;
    T.od_chi_min_pa = QED == SFP_QED_OPTICAL_DEPTH ? pow(10.0, R->od_pair.log_chi_min) : 0.0;
    return T;
}

// photon emission by a massive particle at t (qed/rejection_sampling.py:73-89,
// optical_depth.py:15-62, hard-photon filter cpu.py:226-231).  With the
// learned sampler (optical depth, R->mlp_params) an event returns, instead of
// delta, the uniform u its energy is drawn from, with log10 chi and the
// hard-photon scale hs (1/gamma in float64, gamma in float32); the warp then
// samples delta with the network and applies the cut (sfp_mlp_events).
template <int FORM, int QED>
__device__ __forceinline__ bool sfp_photon_event(const sfp_run_dev* __restrict__ R, const sfp_qed_smem& T,
                                                 const sfp_segment& S, const sfp_instance& I,
                                                 const double* __restrict__ P, double x, double y, double z, double ux,
                                                 double uy, double uz, double t, unsigned int step, long long i,
                                                 double& tau, double& delta, double& hs, double& lchi) {
    using namespace sfp;
    const double dt = R->dt;
    bool ev = false;
    double d = 0.0;
    if (FORM == SFP_FORM_FP64) {
        double F[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (S.push) sfp_field_program(x, y, z, t, P, F);
        const double ig = inv_gamma_massive(ux, uy, uz);
        const double chi = chi_of(F, ux, uy, uz, ig);
        if (QED == SFP_QED_REJECTION) {
            if (chi != 0.0) {
                double r1, r2;
                sfp_step_uniform2(I.seed, S.stream, step, 0u, i, r1, r2);
                ev = photon_event_rs(chi, ig, dt, r1, r2, T.iAt, T.dAt, T.zN, T.zmax, d);
            }
        } else if (R->mlp_params) {
            ev = od_event_u(chi, ig, dt, tau, R->od_photon, T.od_ph, T.od_chi_min_ph, I.seed, S.stream, step, i, d);
            hs = ig;
            lchi = ev ? log10(chi) : 0.0;
        } else {
            ev = od_event(chi, ig, dt, tau, R->od_photon, T.od_ph, T.od_chi_min_ph, I.seed, S.stream, step, i, d);
        }
        if (ev && !(QED == SFP_QED_OPTICAL_DEPTH && R->mlp_params) && d / ig < R->photon_threshold) ev = false;
    } else {
        float F[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (S.push) sfp_field_program32(x, y, z, t, P, F);
        const float g = sfp32::gamma_of(ux, uy, uz, false);
        const float chi = sfp32::chi_of(F, sfp32::d2f(ux), sfp32::d2f(uy), sfp32::d2f(uz), g);
        if (QED == SFP_QED_REJECTION) {
            // straight-line: the draw and the rate for every lane, the
            // conditions combined at the end (chi = 0 gives W = 0)
            float r1, r2;
            sfp_step_uniform2f(I.seed, S.stream, step, 0u, i, r1, r2);
            const float kRate = (float)((kAlpha * kMe) * (kC * kC) / kHbar);
            const float dl = r1 * r1 * r1;
            const float base = __fdividef(dl, (1.0f - dl) * chi);
            const float W = -kRate * sfp32::rate_core(dl * chi, base, T.iAf, T.dAf, T.inv_dzf, T.zN, T.base_maxf, 1.0f);
            ev = (chi > 0.0f) & (r2 < 3.0f * r1 * r1 * W * __fdividef(sfp32::d2f(dt), g)) &
                 !(dl * g < sfp32::d2f(R->photon_threshold));
            d = (double)dl;
        } else {
            // float32 rate lookup, float64 optical depth
            double u = 0.0;
            ev = !((double)chi < T.od_chi_min_ph) &&
                 od_tau_step((double)sfp32::od_rate(chi, R->od_photon, T.od_phf), (double)__fdividef(1.0f, g), dt, tau, I.seed,
                             S.stream, step, i, u);
            if (R->mlp_params) {
                d = u;
                hs = (double)g;
                lchi = ev ? log10((double)chi) : 0.0;
            } else {
                d = ev ? od_bisect((double)chi, u, R->od_photon) : 0.0;
                if (ev && d * (double)g < R->photon_threshold) ev = false;
            }
        }
        if (!ev) d = 0.0;
    }
    delta = d;
    return ev;
}

// pair creation by a photon at t (qed/rejection_sampling.py:92-107,
// optical_depth.py:64-111)
template <int FORM, int QED>
__device__ __forceinline__ bool sfp_pair_event(const sfp_run_dev* __restrict__ R, const sfp_qed_smem& T,
                                               const sfp_segment& S, const sfp_instance& I,
                                               const double* __restrict__ P, double x, double y, double z, double ux,
                                               double uy, double uz, double t, unsigned int step, long long i,
                                               double& tau, double& delta) {
    using namespace sfp;
    const double dt = R->dt;
    bool ev = false;
    double d = 0.0;
    if (FORM == SFP_FORM_FP64) {
        double F[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (S.push) sfp_field_program(x, y, z, t, P, F);
        const double ig = inv_gamma_photon(ux, uy, uz);
        const double chi = chi_of(F, ux, uy, uz, ig);
        if (QED == SFP_QED_REJECTION) {
            if (chi != 0.0 && !(chi < T.chi_pair_min)) {
                double r1, r2;
                sfp_step_uniform2(I.seed, S.stream, step, 0u, i, r1, r2);
                ev = pair_event_rs(chi, ig, dt, r1, r2, T.iAt, T.dAt, T.zN, T.zmax, d);
            }
        } else {
            ev = od_event(chi, ig, dt, tau, R->od_pair, T.od_pa, T.od_chi_min_pa, I.seed, S.stream, step, i, d);
        }
    } else {
        float F[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (S.push) sfp_field_program32(x, y, z, t, P, F);
        // in a zero field (outside every pulse: the far-field cut) chi is
        // exactly 0, so neither method can create a pair or change tau
        const bool field = F[0] != 0.f || F[1] != 0.f || F[2] != 0.f || F[3] != 0.f || F[4] != 0.f || F[5] != 0.f;
        if (field) {
            const float g = sfp32::gamma_of(ux, uy, uz, true);
            const float chi = sfp32::chi_of(F, sfp32::d2f(ux), sfp32::d2f(uy), sfp32::d2f(uz), g);
            if (QED == SFP_QED_REJECTION) {
                if (chi > 0.0f && !((double)chi < T.chi_pair_min)) {
                    float r1, r2;
                    sfp_step_uniform2f(I.seed, S.stream, step, 0u, i, r1, r2);
                    const float kRate = (float)((kAlpha * kMe) * (kC * kC) / kHbar);
                    const float base = __fdividef(1.0f, (r1 * (1.0f - r1)) * chi);
                    const float W =
                        kRate * sfp32::rate_core(chi, base, T.iAf, T.dAf, T.inv_dzf, T.zN, T.base_maxf, -1.0f);
                    ev = r2 < W * __fdividef(sfp32::d2f(dt), g);
                    d = (double)r1;
                }
            } else {
                // float32 rate lookup, float64 optical depth
                double u = 0.0;
                ev = !((double)chi < T.od_chi_min_pa) &&
                     od_tau_step((double)sfp32::od_rate(chi, R->od_pair, T.od_paf), (double)__fdividef(1.0f, g), dt, tau, I.seed,
                                 S.stream, step, i, u);
                d = ev ? od_bisect((double)chi, u, R->od_pair) : 0.0;
            }
        }
        if (!ev) d = 0.0;
    }
    delta = d;
    return ev;
}

// Energies of this warp's emission events from the learned sampler: the
// events are packed into per-warp rows, run through the network 16 rows per
// tensor-core tile (sfp_mlp.cuh), and the hard-photon cut is applied.  On
// entry delta[k] holds each event's uniform u, on exit its delta (0 if cut).
template <int FORM, int ITEMS>
__device__ __forceinline__ void sfp_mlp_events(const sfp_run_dev* __restrict__ R, const sfp_mlp::Smem& M,
                                               bool (&ev)[ITEMS], double (&delta)[ITEMS], const double (&hs)[ITEMS],
                                               const double (&lchi)[ITEMS]) {
    constexpr int NW = SFP_TILE / 32;
    __shared__ float s_x[NW][32 * ITEMS][2];
    __shared__ float s_y[NW][32 * ITEMS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const unsigned int lt = (1u << lane) - 1u;
    int rk[ITEMS];
    int ne = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const unsigned int bal = __ballot_sync(0xffffffffu, ev[k]);
        rk[k] = ne + __popc(bal & lt);
        if (ev[k]) {
            s_x[warp][rk[k]][0] = sfp_mlp::feat_chi(lchi[k]);
            s_x[warp][rk[k]][1] = sfp_mlp::feat_u(delta[k]);
        }
        ne += __popc(bal);
    }
    if (ne == 0) return;
    __syncwarp();
    for (int r0 = 0; r0 < ne; r0 += 16) {
        float x0[2], x1[2], y[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = r0 + g + 8 * h;
            x0[h] = r < ne ? s_x[warp][r][0] : 0.0f;
            x1[h] = r < ne ? s_x[warp][r][1] : 0.0f;
        }
        sfp_mlp::tile16(M, x0, x1, y);
        if (t == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + g + 8 * h;
                if (r < ne) s_y[warp][r] = y[h];
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (!ev[k]) continue;
        const double d = sfp_mlp::delta_of(s_y[warp][rk[k]]);
        const bool cut = FORM == SFP_FORM_FP64 ? d / hs[k] < R->photon_threshold : d * hs[k] < R->photon_threshold;
        ev[k] = !cut;
        delta[k] = cut ? 0.0 : d;
    }
    __syncwarp();
}

// largest j with start[j] <= tk (binary search over a group's tile starts)
__device__ __forceinline__ int sfp_find_group_pos(const long long* __restrict__ start, int n, long long tk) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (start[mid] <= tk) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// The end of a step's event kernels (sfp_step_end), one block of 256 threads:
//   scan    -- an exclusive scan of both groups' super-tile event counts in
//              tile order, restarted at each instance and kept per append
//              channel, so super_pre[s] is the number of children that the
//              same instance's earlier segments and tiles with the same
//              destinations append before super-tile s; every segment's
//              events become its destinations' append counts, and if a
//              destination lacks room for the step's children the step
//              waits for the host (append_wait) with nothing changed;
//   fold    -- the appends enter n_buffered, t and step advance;
//   prepare -- each group's tile length and tile map for the next step,
//              tickets, super-tile counts at zero.
// The next step's plan goes to the other of two slots (st->plan, tile_start,
// n_buf_step; st->cur then names it), as the appends kernel that follows
// still works by the plan of the step that ran.
//
// It runs in the block that finishes last of the step's last event launch
// (sfp_last_block).  As two launches of one block each, the scan and the
// bookkeeping took 7 and 5 us of a small step (1e4 e-), most of it chains of
// dependent loads, and two launch gaps of 2 us; here the segments' and the
// steps' data are loaded at once and held in shared memory.
// sfp_book_kernel prepares the first step of a call and folds a resumed one.
// ---------------------------------------------------------------------------
#define SFP_PREP 1
// the next step's massive / photon launch is the long-tile kernel, so that
// group's tiles must be SFP_TILE_MAX long
#define SFP_PREP_M 2
#define SFP_PREP_P 4
#define SFP_FOLD 8
#define SFP_SCAN 16
// (sfp_book_kernel) the call keeps a store of hot photons, which is built next
#define SFP_HOT 32
// the next step runs in the one-launch kernel, with flags >> SFP_SMALL_SHIFT warps
#define SFP_SMALL 64
#define SFP_SMALL_SHIFT 8

// a step as its kernels see it
struct sfp_step_view {
    double t, lag;  // lag: steps since the stored photon positions
    long long step, n_mtiles, n_ptiles;
    const long long *m_start, *p_start, *n_buf;
    int mtile, ptile;
};
SFP_DEVICE_INLINE sfp_step_view sfp_view(const sfp_run_dev* __restrict__ R, int slot) {
    const sfp_step_state* st = R->st;
    const sfp_step_plan& p = st->plan[slot];
    sfp_step_view v;
    v.t = p.t;
    v.step = p.step;
    v.lag = (double)(p.step - st->pos_epoch);
    v.n_mtiles = p.n_mtiles;
    v.n_ptiles = p.n_ptiles;
    v.mtile = p.mtile;
    v.ptile = p.ptile;
    v.m_start = R->mg.tile_start + slot * (R->mg.n_seg + 1);
    v.p_start = R->pg.tile_start + slot * (R->pg.n_seg + 1);
    v.n_buf = R->n_buf_step + slot * R->n_seg;
    return v;
}

// true in every thread of the block that is last to arrive of the launch's
// `blocks`; earlier blocks' writes are then visible to it
__device__ __forceinline__ bool sfp_last_block(sfp_step_state* st, unsigned int blocks) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const int n = atomicAdd(&st->blocks_done, 1);
        s_last = n == (int)blocks - 1;
        if (s_last) st->blocks_done = 0;
    }
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

SFP_DEVICE_INLINE long long sfp_warp_sum64(long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

SFP_DEVICE_INLINE uint4 shfl_up_u4(uint4 v, int o) {
    return uint4{__shfl_up_sync(0xffffffffu, v.x, o), __shfl_up_sync(0xffffffffu, v.y, o),
                 __shfl_up_sync(0xffffffffu, v.z, o), __shfl_up_sync(0xffffffffu, v.w, o)};
}

// inclusive warp scan of (head, value) pairs: a head restarts the sum
SFP_DEVICE_INLINE void seg_scan_warp(unsigned int& h, uint4& v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int oh = __shfl_up_sync(0xffffffffu, h, o);
        const uint4 ov = shfl_up_u4(v, o);
        if (lane >= o) {
            if (!h) v = sfp::u4_add(ov, v);
            h |= oh;
        }
    }
}

// tiles of pt particles (a multiple of 32) that n particles take
SFP_DEVICE_INLINE long long sfp_tiles_of(long long n, int pt) {
    if ((n >> 31) == 0) return (long long)(((unsigned int)n + (unsigned int)pt - 1u) / (unsigned int)pt);
    return (n + pt - 1) / pt;
}

// the group's tile map for tiles of pt particles, by a warp, from the next
// step's counts nb: each segment's tiles start at a multiple of
// SFP_SUPER_TILE; returns the number of tiles
SFP_DEVICE_INLINE long long sfp_group_map(const int* seg, int n_seg, const long long* nb, int pt, long long* start) {
    const int lane = threadIdx.x & 31;
    long long carry = 0, end = 0;
    for (int j0 = 0; j0 < n_seg; j0 += 32) {
        const int j = j0 + lane;
        const long long t = j < n_seg ? sfp_tiles_of(nb[seg[j]], pt) : 0;
        const long long own = (t + SFP_SUPER_TILE - 1) / SFP_SUPER_TILE * SFP_SUPER_TILE;
        long long inc = own;
        __syncwarp();
        for (int o = 1; o < 32 && o < n_seg - j0; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        const long long at = carry + inc - own;
        if (j < n_seg) start[j] = at;
        const int last = min(31, n_seg - 1 - j0);
        __syncwarp();
        end = __shfl_sync(0xffffffffu, at + t, last);
        carry += __shfl_sync(0xffffffffu, inc, last);
    }
    if (lane == 0) start[n_seg] = end;
    __syncwarp();
    return end;
}

// a group's population, by a warp
SFP_DEVICE_INLINE long long sfp_group_count(const int* seg, int n_seg, const long long* nb) {
    long long n = 0;
    for (int j = threadIdx.x & 31; j < n_seg; j += 32) n += nb[seg[j]];
    __syncwarp();
    for (int o = 1; o < 32 && o < n_seg; o <<= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    return __shfl_sync(0xffffffffu, n, 0);
}

// the group's tile of the next step (SFP_TILE_MIN..SFP_TILE_MAX, a power of
// two), for n particles in at most `target` tiles
SFP_DEVICE_INLINE int sfp_tile_rule(long long n, long long target) {
    int pt = SFP_TILE_MIN;
    while (pt < SFP_TILE_MAX && pt * target < n) pt <<= 1;
    return pt;
}

// The one-launch kernel's tiles: about one per warp, so that no warp takes a
// second one while others are done.  A warp's 32 e+- take several times as long
// as its 32 photons (weight), so the tiles' lengths are the shares of that
// sum; both are multiples of 32, not powers of two (1e4 e- and 1.4e5 photons:
// tiles of 32 and 64 left 13 % of the warps a second tile).  Weights measured:
// rejection sampling 3 (1e5 e-, 1.2e6 photons, float32 form: 37.0 us a step,
// with 5 38.4, with 8 39.9), optical depth 8 (1e5 e+-, 8e5 photons: 186 us,
// with 5 203, with 3 236).
SFP_DEVICE_INLINE int sfp_small_tile(long long m, long long p, int warps, bool massive, int weight) {
    const long long work = weight * ((m + 31) >> 5) + ((p + 31) >> 5);  // in sub-steps of photons
    const int share = (int)min((long long)(SFP_TILE_MAX / 32), (work + warps - 1) / warps);
    const int sub = massive ? (share + weight - 1) / weight : share;
    return 32 * (sub < 1 ? 1 : sub);
}

// What both halves of a step's end share: the counts and appends of every
// segment, in shared memory (or the run's scratch)
struct sfp_end_data {
    sfp_end_seg* seg;
    unsigned long long* app;
    long long* nb;
};
SFP_DEVICE_INLINE sfp_end_data sfp_end_arrays(const sfp_run_dev* __restrict__ R, sfp_end_smem& Q) {
    const bool held = R->n_seg <= SFP_END_SEGS;
    return sfp_end_data{held ? Q.seg : R->end_seg, held ? Q.app : R->end_app, held ? Q.nb : R->end_nb};
}

// loads the step's counts, and (SFP_SCAN) scans its events; false if a
// destination lacks room
__device__ __forceinline__ bool sfp_end_scan(const sfp_run_dev* __restrict__ R, int flags, sfp_end_smem& Q) {
    sfp_step_state* st = R->st;
    const int n = R->n_seg, nm = R->mg.n_seg, np = R->pg.n_seg;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const sfp_end_data E = sfp_end_arrays(R, Q);
    sfp_end_seg* const seg = E.seg;
    unsigned long long* const app = E.app;
    long long* const nb = E.nb;
    const int cur = st->cur;
    const long long n_mtiles = st->plan[cur].n_mtiles, n_ptiles = st->plan[cur].n_ptiles;
    const long long *m_start = R->mg.tile_start + cur * (nm + 1), *p_start = R->pg.tile_start + cur * (np + 1);
    const long long* n_buf = R->n_buf_step + cur * n;
    __syncthreads();  // the dynamic shared memory's earlier users are done
    if (threadIdx.x == 0) Q.lacks = 0;
    const int nsm = (int)((n_mtiles + SFP_SUPER_TILE - 1) / SFP_SUPER_TILE);
    const int nsp = (int)((n_ptiles + SFP_SUPER_TILE - 1) / SFP_SUPER_TILE);
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        nb[k] = (flags & SFP_FOLD) ? n_buf[k] : __ldcg(&R->n_buffered[k]);
        app[k] = (flags & (SFP_FOLD | SFP_SCAN)) == SFP_FOLD ? __ldcg(&R->appended[k]) : 0ull;
        if (flags & SFP_SCAN) {  // entry k of the massive group's segments, then the photon group's
            const bool massive = k < nm;
            const int j = massive ? k : k - nm;
            const sfp_segment& S = R->seg[massive ? R->mg.seg[j] : R->pg.seg[j]];
            sfp_end_seg e;
            e.super0 = massive ? (int)(m_start[j] / SFP_SUPER_TILE) : nsm + (int)(p_start[j] / SFP_SUPER_TILE);
            e.chain = 2 * S.instance + (massive ? 0 : 1);
            e.channel = S.channel;
            e.dest0 = massive ? S.photon_dest : S.ele_dest;
            e.dest1 = massive ? -1 : S.pos_dest;
            seg[k] = e;
        }
    }
    __syncthreads();
    if (flags & SFP_SCAN) {
        // the super-tiles of both groups as one sequence, a run of them per
        // thread; a head is the first super-tile of its instance and group
        const int ns = nsm + nsp;
        const int per = (ns + (int)blockDim.x - 1) / (int)blockDim.x;
        const int s0 = min(ns, (int)threadIdx.x * per), s1 = min(ns, s0 + per);
        auto count = [&](int s) { return __ldcg(s < nsm ? &R->mg.super_cnt[s] : &R->pg.super_cnt[s - nsm]); };
        // the last entry that starts at or before s
        auto find = [&](int s) {
            int lo = 0, hi = n - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (seg[mid].super0 <= s) lo = mid;
                else hi = mid - 1;
            }
            return lo;
        };
        unsigned int h = 0, c0 = 0;
        uint4 v{0u, 0u, 0u, 0u};
        int j0 = 0, before = -1;  // the run's first entry; the chain of the super-tile before it
        if (s0 < s1) {
            c0 = count(s0);
            j0 = find(s0);
            if (s0 > 0) before = s0 - 1 >= seg[j0].super0 ? seg[j0].chain : seg[find(s0 - 1)].chain;
            int j = j0, prev = before;
            for (int s = s0; s < s1; ++s) {
                while (j + 1 < n && seg[j + 1].super0 <= s) ++j;
                if (seg[j].chain != prev) {
                    h = 1;
                    v = uint4{0u, 0u, 0u, 0u};
                    prev = seg[j].chain;
                }
                v = sfp::u4_add(v, sfp::u4_one(seg[j].channel, s == s0 ? c0 : count(s)));
            }
        }
        __syncwarp();  // the lanes' runs differ in length: together again before the shuffles
        seg_scan_warp(h, v);
        if (lane == 31) {
            Q.wh[warp] = h;
            Q.wv[warp] = v;
        }
        __syncthreads();
        // exclusive value of this thread: earlier warps, then earlier lanes of this warp
        unsigned int lh = __shfl_up_sync(0xffffffffu, h, 1);
        uint4 run = shfl_up_u4(v, 1);
        if (lane == 0) {
            lh = 0u;
            run = uint4{0u, 0u, 0u, 0u};
        }
        for (int w = warp - 1; w >= 0 && !lh; --w) {
            run = sfp::u4_add(Q.wv[w], run);
            lh = Q.wh[w];
        }
        if (s0 < s1) {
            int j = j0, prev = before;
            unsigned long long acc = 0ull;
            auto add = [&]() {
                if (!acc) return;
                if (seg[j].dest0 >= 0) atomicAdd(&app[seg[j].dest0], acc);
                if (seg[j].dest1 >= 0) atomicAdd(&app[seg[j].dest1], acc);
                acc = 0ull;
            };
            for (int s = s0; s < s1; ++s) {
                while (j + 1 < n && seg[j + 1].super0 <= s) {
                    add();
                    ++j;
                }
                if (seg[j].chain != prev) {
                    run = uint4{0u, 0u, 0u, 0u};
                    prev = seg[j].chain;
                }
                const unsigned int c = s == s0 ? c0 : count(s);
                (s < nsm ? R->mg.super_pre[s] : R->pg.super_pre[s - nsm]) = (long long)sfp::u4_get(run, seg[j].channel);
                run = sfp::u4_add(run, sfp::u4_one(seg[j].channel, c));
                acc += c;
            }
            add();
        }
        __syncthreads();  // every append count is in
        // exact room check: the appends kernel writes nothing unless every
        // destination holds its children; otherwise the step waits for the host
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            R->appended[k] = app[k];
            if (app[k] && nb[k] + (long long)app[k] > R->seg[k].capacity) Q.lacks = 1;
        }
        __syncthreads();
        if (Q.lacks) {
            if (threadIdx.x == 0) {
                st->append_wait = 1;
                st->halted = 1;
            }
            return false;
        }
    }
    return true;
}

// folds the step (SFP_FOLD) and prepares the next one (SFP_PREP); nb and app
// as sfp_end_scan left them.  small: the tiles of the one-launch kernel, whose
// warps it names, or 0
__device__ __forceinline__ void sfp_end_plan(const sfp_run_dev* __restrict__ R, int flags, sfp_end_smem& Q, int small) {
    sfp_step_state* st = R->st;
    const int n = R->n_seg, nm = R->mg.n_seg, np = R->pg.n_seg;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const sfp_end_data E = sfp_end_arrays(R, Q);
    unsigned long long* const app = E.app;
    long long* const nb = E.nb;
    const int cur = st->cur, slot = (flags & SFP_FOLD) ? cur ^ 1 : cur;
    const double t = (flags & SFP_FOLD) ? st->plan[cur].t + R->dt : st->t;
    const long long step = (flags & SFP_FOLD) ? st->plan[cur].step + 1 : st->step;
    const bool go = !(st->halted || st->error || st->append_wait);
    if (flags & SFP_FOLD) {
        long long ps = 0;
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            ps += nb[k];
            nb[k] += (long long)app[k];
            R->n_buffered[k] = nb[k];
            R->appended[k] = 0ull;
        }
        __syncwarp();
        ps = sfp_warp_sum64(ps);
        if (lane == 0) Q.ps[warp] = ps;
    }
    __syncthreads();
    if ((flags & SFP_PREP) && go && warp < 2) {
        const int* seg_m = R->mg.seg;
        const int* seg_p = R->pg.seg;
        const bool massive = warp == 0;
        const int* seg = massive ? seg_m : seg_p;
        const int ns = massive ? nm : np;
        long long* start = massive ? R->mg.tile_start + slot * (nm + 1) : R->pg.tile_start + slot * (np + 1);
        const long long most = massive ? R->mg.max_tiles : R->pg.max_tiles;
        int pt;
        if (small)
            pt = sfp_small_tile(sfp_group_count(seg_m, nm, nb), sfp_group_count(seg_p, np, nb), small, massive,
                                R->qed == SFP_QED_REJECTION ? 3 : 8);
        else
            pt = sfp_tile_rule(sfp_group_count(seg, ns, nb), massive ? SFP_TILE_TARGET_M : SFP_TILE_TARGET);
        // a map too long for the counters takes a longer tile
        long long tiles = sfp_group_map(seg, ns, nb, pt, start);
        while (tiles > most && pt < SFP_TILE_MAX) {
            pt = min(2 * pt, SFP_TILE_MAX);
            tiles = sfp_group_map(seg, ns, nb, pt, start);
        }
        if (lane == 0) {
            Q.tiles[warp] = tiles;
            Q.tile[warp] = pt;
        }
    }
    if ((flags & SFP_PREP) && go)
        for (int k = threadIdx.x; k < n; k += blockDim.x) R->n_buf_step[slot * n + k] = nb[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        if (flags & SFP_FOLD) {
            long long all = 0;
            for (int w = 0; w < 8; ++w) all += Q.ps[w];
            st->particle_steps += all;
            st->t = t;
            st->step = step;
            st->cur = slot;
        }
        if ((flags & SFP_PREP) && !go) st->skip = 1;
    }
    if (!(flags & SFP_PREP) || !go) return;
    const long long m_tiles = Q.tiles[0], p_tiles = Q.tiles[1];
    const int mt = Q.tile[0], pt = Q.tile[1];
    int error = SFP_DEV_OK;
    if (m_tiles > R->mg.max_tiles || p_tiles > R->pg.max_tiles) error = SFP_DEV_CAPACITY;
    else if (((flags & SFP_PREP_M) && mt != SFP_TILE_MAX) || ((flags & SFP_PREP_P) && pt != SFP_TILE_MAX))
        error = SFP_DEV_TILE;  // the long-tile kernels launched for a step with shorter tiles
    if (threadIdx.x == 0) {
        if (error != SFP_DEV_OK) {
            st->error = error;
            st->skip = 1;
        } else {
            sfp_step_plan& P = st->plan[slot];
            P.t = t;
            P.step = step;
            P.n_mtiles = m_tiles;
            P.n_ptiles = p_tiles;
            P.mtile = mt;
            P.ptile = pt;
            st->mticket = 0;
            st->pticket = 0;
            st->skip = 0;
        }
    }
    if (error != SFP_DEV_OK) return;
    // the group kernels add into the super-tile counts: start them at zero
    const long long zm = (m_tiles + SFP_SUPER_TILE - 1) / SFP_SUPER_TILE;
    const long long zp = (p_tiles + SFP_SUPER_TILE - 1) / SFP_SUPER_TILE;
    for (long long k = threadIdx.x; k < zm; k += blockDim.x) R->mg.super_cnt[k] = 0u;
    for (long long k = threadIdx.x; k < zp; k += blockDim.x) R->pg.super_cnt[k] = 0u;
}

__device__ __forceinline__ void sfp_step_end(const sfp_run_dev* __restrict__ R, int flags, sfp_end_smem& Q) {
    if (sfp_end_scan(R, flags, Q)) sfp_end_plan(R, flags, Q, (flags & SFP_SMALL) ? flags >> SFP_SMALL_SHIFT : 0);
}

extern "C" __global__ void __launch_bounds__(256) sfp_book_kernel(const sfp_run_dev* __restrict__ R, int flags) {
    extern __shared__ __align__(16) double s_tab[];
    if (flags & SFP_PREP) {
        if (threadIdx.x == 0) R->st->hot_ok = (flags & SFP_HOT) ? 1 : 0;
        if (flags & SFP_HOT)
            for (int k = threadIdx.x; k < R->n_seg; k += blockDim.x) R->hot.count[k] = 0ull;
    }
    sfp_step_end(R, flags, *reinterpret_cast<sfp_end_smem*>(s_tab));
}

// what a launch does once its blocks are done (`tail`: sfp_step_end's flags,
// or 0), in the last of them; `scratch`: its dynamic shared memory.  Every
// block of the grid comes here, those without tiles at once: a block may start
// after the others are done (another stream's kernels hold the SMs), and if the
// step's end did not wait for it, it would read the next step's plan and take
// that step's tiles before this step's children are written.  The idle blocks'
// arrivals cost nothing that shows: 64 collisions, 1e6 e- and 1.2e7 photons, 32
// steps, 7.05 ms with the busy blocks' arrivals alone, 7.04 with all.
__device__ __noinline__ void sfp_tail(const sfp_run_dev* __restrict__ R, int tail, void* scratch) {
    if (!tail || !sfp_last_block(R->st, gridDim.x)) return;
    sfp_step_end(R, tail, *static_cast<sfp_end_smem*>(scratch));
}

// blocks of a group launch that have tiles to take, of `grid`: one for four
// tiles (the others go to the launch's tail at once)
SFP_DEVICE_INLINE unsigned int sfp_busy_blocks(long long n_tiles, unsigned int grid) {
    const long long b = (n_tiles + 3) / 4;
    return b < 1 ? 1u : b < (long long)grid ? (unsigned int)b : grid;
}

// ---------------------------------------------------------------------------
// The copy ring of both group kernels.  A warp streams its tile (32 to 1024
// particles) 32 at a time through STAGES shared-memory stages
// filled with cp.async, so the state of the next sub-steps is in flight
// while the current one computes.  The copies and the stores address the
// tile through a per-warp descriptor in shared memory, written once per
// tile: slots 0..NC-1 the staged float64 arrays (x, y, z, ux, uy, uz, then
// tau under optical depth, then sx, sy, sz for spin), slot NC the pruned
// flags, slot NC+1 the delta array; each offset to the tile's first
// particle (NULL where the segment has no such array).
// ---------------------------------------------------------------------------
template <int NC>
struct sfp_ring {
    static constexpr int STAGE_BYTES = NC * 32 * 8 + 32;  // NC components + 32 flags
};

template <int QED, bool SPIN>
SFP_DEVICE_INLINE char* sfp_desc_slot(const sfp_segment& S, int c, long long base) {
    constexpr int OD = QED == SFP_QED_OPTICAL_DEPTH ? 1 : 0;
    constexpr int NC = 6 + OD + (SPIN ? 3 : 0);
    double* p = nullptr;
    switch (c) {
        case 0: p = S.x; break;
        case 1: p = S.y; break;
        case 2: p = S.z; break;
        case 3: p = S.ux; break;
        case 4: p = S.uy; break;
        case 5: p = S.uz; break;
        default: break;
    }
    if (OD && c == 6) p = S.tau;
    if (SPIN && c == 6 + OD) p = S.sx;
    if (SPIN && c == 7 + OD) p = S.sy;
    if (SPIN && c == 8 + OD) p = S.sz;
    if (c == NC) return reinterpret_cast<char*>(S.pruned + base);
    if (c == NC + 1) p = S.delta;
    return p ? reinterpret_cast<char*>(p + base) : nullptr;
}

// copies of sub-step `sub` (tile particles 32 sub .. + 31) into one stage:
// copy c is component c/16 of particles 2(c%16), +1 (c < 16 NC) or 16
// flags, always to dst + 16 c, so components land at dst + 256 comp and the
// flags at dst + 256 NC.  `left` = particles of the segment from the tile's
// first on; entries past them are zero-filled and not read.  One commit group.
// Every segment has components 0-5 (x .. uz) and, in the spin variant, the
// spin components; only component 6 under optical depth (tau) can be absent,
// so only copies that can read it test for a NULL array (at compile time
// for the others: copy c = lane + 32 k reads components 2k and 2k + 1).
template <int NC, int OD>
__device__ __forceinline__ void sfp_ring_issue(char* const* D, int sub, long long left, unsigned char* dst,
                                               int lane) {
    constexpr int NCOPY = NC * 16 + 2;
    const bool full = left >= (long long)(sub + 1) * 32;  // warp-uniform: no copy is short
#pragma unroll
    for (int k = 0; k < (NCOPY + 31) / 32; ++k) {
        const int c = lane + 32 * k;
        if (c < NC * 16) {
            const int e = sub * 32 + 2 * (c & 15);
            const char* src = D[c >> 4];
            unsigned int nb = 16u;
            if (!full) nb = left - e >= 2 ? 16u : (left - e == 1 ? 8u : 0u);
            if (OD && 2 * k <= 6 && 6 <= 2 * k + 1 && !src) nb = 0u;  // the segment has no tau array
            sfp::cp_async16(dst + c * 16, nb ? (const void*)(src + (size_t)e * 8) : (const void*)D[NC], nb);
        } else if (c < NCOPY) {
            const int e = sub * 32 + 16 * (c - NC * 16);
            const char* src = D[NC];
            unsigned int nb = 16u;
            if (!full) nb = left - e >= 16 ? 16u : (left - e > 0 ? (unsigned int)(left - e) : 0u);
            sfp::cp_async16(dst + c * 16, nb ? (const void*)(src + e) : (const void*)src, nb);
        }
    }
    sfp::cp_async_commit();
}

// The copies of a full tile (no copy is short): copy c = lane + 32 k of
// sub-step `sub` reads component c / 16 at byte offset 256 sub + 16 (c % 16)
// of the tile (or the flags at 32 sub + 16 (c - 16 NC)), straight from the
// descriptor, with none of the general issue's bounds arithmetic; a
// component the segment lacks is zero-filled.
template <int NC, int OD>
__device__ __forceinline__ void sfp_ring_issue_full(char* const* D, int sub, unsigned char* dst, int lane) {
    constexpr int NCOPY = NC * 16 + 2;
    const unsigned int off = (unsigned int)sub * 256u + 16u * (unsigned int)(lane & 15);
#pragma unroll
    for (int k = 0; k < (NCOPY + 31) / 32; ++k) {
        const int c = lane + 32 * k;
        if (c < NC * 16) {
            const char* p = D[c >> 4];
            const bool has = !(OD && 2 * k <= 6 && 6 <= 2 * k + 1) || p != nullptr;  // see sfp_ring_issue
            sfp::cp_async16(dst + c * 16, has ? (const void*)(p + off) : (const void*)D[NC], has ? 16u : 0u);
        } else if (c < NCOPY) {
            sfp::cp_async16(dst + c * 16, D[NC] + sub * 32 + 16 * (c - NC * 16), 16u);
        }
    }
    sfp::cp_async_commit();
}

// ---------------------------------------------------------------------------
// Massive group.  Each warp takes tiles of the step's length by ticket
// (the next ticket in flight while the tile computes) and streams them
// through the copy ring; after the tables are staged no block barrier is
// taken.  Per particle: the photon event at t (rejection sampling or optical
// depth, hard-photon cut); an emitter is marked (pruned = SFP_MARK) with its
// delta stored and keeps its state at t for the appends kernel; every other
// alive particle is pushed to t+dt (Boris / Boris-TBMT, LL/CLL) and stored.
// The warp's event count goes to its tile's counter and its super-tile's.
// ---------------------------------------------------------------------------
template <int FORM, int QED, int STAGES, bool SPIN, bool LONG>
__device__ __forceinline__ unsigned int sfp_massive_tile(const sfp_run_dev* __restrict__ R, const sfp_qed_smem& T,
                                                         const sfp_mlp::Smem& M, const sfp_segment& S_in, char** desc,
                                                         unsigned char* ring, int SB, int PT, long long base,
                                                         long long left, double t, double dt, unsigned int step) {
    using namespace sfp;
    // a copy: what depends on the segment alone (the float64 push's factors, two
    // divisions) is formed once per tile, as no store can change it
    const sfp_segment S = S_in;
    constexpr int OD = QED == SFP_QED_OPTICAL_DEPTH ? 1 : 0;
    constexpr int NC = 6 + OD + (SPIN ? 3 : 0);
    const int lane = threadIdx.x & 31;
    const sfp_instance& I = R->inst[S.instance];
    const double* __restrict__ P = sfp_field_params(I);
    const bool rad = S.radiating != 0, push = S.push != 0;
    const sfp_pc32 K32 = push_consts32(S, t, dt);  // float32 form's push constants of this segment
    __syncwarp();  // the previous tile's lanes are done with the descriptor and the stages
    if (lane < NC + 2) desc[lane] = sfp_desc_slot<QED, SPIN>(S, lane, base);
    __syncwarp();
    char* const* D = desc;
    unsigned int cnt = 0;
    // LONG: a tile of SFP_TILE_MAX particles, 32 sub-steps of 32 with
    // compile-time bounds; else the step's shorter tile, sub-steps up to its
    // last particle (`len`, the tile length or fewer at a segment's end)
    const int len = LONG ? SFP_TILE_MAX : (int)min(left, (long long)PT);
    const bool full = LONG ? left >= (long long)SFP_TILE_MAX : len == PT;
    auto issue = [&](int sb, unsigned char* dst) {
        if (full) sfp_ring_issue_full<NC, OD>(D, sb, dst, lane);
        else sfp_ring_issue<NC, OD>(D, sb, LONG ? left : (long long)len, dst, lane);
    };
#pragma unroll
    for (int k = 0; k < STAGES - 1; ++k) {
        if (LONG || 32 * k < len) issue(k, ring + k * SB);
        else cp_async_commit();  // a short tile: nothing to fetch, the group count stays
    }
#pragma unroll 1
    // rd: the stage of `sub` (sub % STAGES); the stage refilled, that of
    // sub + STAGES - 1, is the one before it
    for (int sub = 0, rd = 0; LONG ? sub < SFP_TILE_MAX / 32 : 32 * sub < len;
         ++sub, rd = rd == STAGES - 1 ? 0 : rd + 1) {
        __syncwarp();  // every lane has read the stage about to be refilled
        const int nsub = sub + STAGES - 1;
        if (LONG ? nsub < SFP_TILE_MAX / 32 : 32 * nsub < len)
            issue(nsub, ring + (rd == 0 ? STAGES - 1 : rd - 1) * SB);
        else
            cp_async_commit();
        cp_async_wait<STAGES - 1>();
        __syncwarp();  // the stage of `sub` is complete for the whole warp
        const unsigned char* stg = ring + rd * SB;
        const double* sd = reinterpret_cast<const double*>(stg);
        const int e = sub * 32 + lane;  // particle index from the tile's first
        const long long i = base + e;
        const bool alive = (LONG ? e < left : e < len) && stg[NC * 256 + lane] == 0;
        double x = sd[lane], y = sd[32 + lane], z = sd[64 + lane];
        double ux = sd[96 + lane], uy = sd[128 + lane], uz = sd[160 + lane];
        double tau = OD ? sd[192 + lane] : 0.0;
        double sx = 0.0, sy = 0.0, sz = 0.0;
        if (SPIN) {
            sx = sd[(6 + OD) * 32 + lane];
            sy = sd[(7 + OD) * 32 + lane];
            sz = sd[(8 + OD) * 32 + lane];
        }
        // every lane runs the event test and the push (dead lanes on their
        // zero-filled stage entries); marks and stores are conditional
        bool ev = false;
        double delta = 0.0, hs = 0.0, lchi = 0.0;
        if (rad) {
            const bool e1 = sfp_photon_event<FORM, QED>(R, T, S, I, P, x, y, z, ux, uy, uz, t, step, i, tau, delta, hs,
                                                        lchi);
            ev = alive & e1;
        }
        if (OD && R->mlp_params) {  // warp-uniform: the learned sampler draws the events' energies
            bool e1[1] = {ev};
            double d1[1] = {delta};
            const double h1[1] = {hs}, l1[1] = {lchi};
            sfp_mlp_events<FORM, 1>(R, M, e1, d1, h1, l1);
            ev = e1[0];
            delta = d1[0];
        }
        if (ev) {
            // the appends kernel writes the photon and pushes the parent
            reinterpret_cast<unsigned char*>(D[NC])[e] = SFP_MARK;
            reinterpret_cast<double*>(D[NC + 1])[e] = delta;
        }
        if (FORM == SFP_FORM_FP64) push_massive(x, y, z, ux, uy, uz, sx, sy, sz, S, P, t, dt);
        else push_massive32<false>(x, y, z, ux, uy, uz, sx, sy, sz, S, P, K32);
        if (!ev && alive && push) {
            reinterpret_cast<double*>(D[0])[e] = x;
            reinterpret_cast<double*>(D[1])[e] = y;
            reinterpret_cast<double*>(D[2])[e] = z;
            reinterpret_cast<double*>(D[3])[e] = ux;
            reinterpret_cast<double*>(D[4])[e] = uy;
            reinterpret_cast<double*>(D[5])[e] = uz;
            if (SPIN) {
                reinterpret_cast<double*>(D[6 + OD])[e] = sx;
                reinterpret_cast<double*>(D[7 + OD])[e] = sy;
                reinterpret_cast<double*>(D[8 + OD])[e] = sz;
            }
        }
        if (OD && alive && rad && D[6]) reinterpret_cast<double*>(D[6])[e] = tau;
        cnt += __popc(__ballot_sync(0xffffffffu, ev));
    }
    return cnt;
}

// LONG: the kernel of steps whose tiles are all SFP_TILE_MAX long (the host
// launches it while the group's population guarantees that, and the
// bookkeeping kernel refuses a step planned otherwise with SFP_DEV_TILE).
template <int FORM, int QED, int STAGES, bool LONG>
__device__ __forceinline__ void sfp_massive_body(const sfp_run_dev* __restrict__ R, int tail) {
    using namespace sfp;
    constexpr int OD = QED == SFP_QED_OPTICAL_DEPTH ? 1 : 0;
    extern __shared__ __align__(16) double s_tab[];
    __shared__ char* s_desc[SFP_TILE / 32][6 + OD + 3 + 2];
    sfp_step_state* st = R->st;
    if (st->skip || st->halted) return;
    const sfp_step_view V = sfp_view(R, st->cur);
    const long long n_tiles = V.n_mtiles;
    const unsigned int busy = sfp_busy_blocks(n_tiles, gridDim.x);
    if (blockIdx.x >= busy) {
        sfp_tail(R, tail, s_tab);
        return;
    }
    if (st->hot_ok)  // the hot photons' events are added to the photon tiles' counts
        for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < V.n_ptiles;
             k += (long long)busy * blockDim.x)
            R->pg.tile_cnt[k] = 0u;
    if (n_tiles == 0) {
        sfp_tail(R, tail, s_tab);
        return;
    }
    const int PT = LONG ? SFP_TILE_MAX : V.mtile;
    const double t = V.t;
    const double dt = R->dt;
    const unsigned int step = (unsigned int)V.step;
    const sfp_qed_smem T = sfp_stage_tables<FORM, QED>(R, s_tab);
    // learned photon-energy sampler: weights after the tables
    sfp_mlp::Smem& M = *reinterpret_cast<sfp_mlp::Smem*>(reinterpret_cast<unsigned char*>(s_tab) + R->mlp_off);
    if (OD && R->mlp_params) sfp_mlp::stage(M, R->mlp_params);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int SB = R->m_stage_bytes;
    unsigned char* ring = reinterpret_cast<unsigned char*>(s_tab) + R->m_ring_off + (size_t)warp * STAGES * SB;

    int tk = 0;
    if (lane == 0) tk = atomicAdd(&st->mticket, 1);
    long long tile = __shfl_sync(0xffffffffu, tk, 0);
    while (tile < n_tiles) {
        if (lane == 0) tk = atomicAdd(&st->mticket, 1);  // next ticket, in flight during this tile
        const int pos = sfp_find_group_pos(V.m_start, R->mg.n_seg, tile);
        const sfp_segment& S = R->seg[R->mg.seg[pos]];
        const long long N = V.n_buf[R->mg.seg[pos]];
        const long long base = (tile - V.m_start[pos]) * (long long)PT;
        unsigned int cnt = 0;
        if (base < N) {  // else: alignment padding between segments
            if (S.spin)
                cnt = sfp_massive_tile<FORM, QED, STAGES, true, LONG>(R, T, M, S, s_desc[warp], ring, SB, PT, base,
                                                                      N - base, t, dt, step);
            else
                cnt = sfp_massive_tile<FORM, QED, STAGES, false, LONG>(R, T, M, S, s_desc[warp], ring, SB, PT, base,
                                                                       N - base, t, dt, step);
        }
        if (lane == 0) {
            R->mg.tile_cnt[tile] = cnt;
            if (cnt) atomicAdd(&R->mg.super_cnt[tile / SFP_SUPER_TILE], cnt);
        }
        tile = __shfl_sync(0xffffffffu, tk, 0);
    }
    sfp_tail(R, tail, s_tab);
}

// ---------------------------------------------------------------------------
// Photon group.  Same tiles, tickets and ring.  Per photon: the position at
// t (stored position + (step - pos_epoch) pushes, photon_shift), the pair
// event at t; a converted photon is marked (pruned = SFP_MARK, not pushed)
// and its delta stored for the appends kernel.  A photon that does not
// convert writes nothing: its push is the epoch's advance, so the kernel
// reads 49 bytes per photon (state and flag) and writes only events.
//
// Rejection sampling: an event needs r2 < W(r1) dt / gamma, and r2 is never
// below 2^-33 (float32 draws) or 2^-53 (float64 draws).  The pair-rate bound
// of the photon's chi bin (R->pair_bound) times dt / gamma below that means
// no draw passes: the photon is done at once, with no draw and no rate.
// Before any field is evaluated, a photon's energy alone bounds its chi
// (chi <= gamma (|E| + c|B|)_max / E_s, sfp_pair_reachable): most photons
// of a cascade are too soft for any draw to pass anywhere in the pulse and
// are done after reading their momentum.  The others go, with their stored
// state, to a 32-entry per-warp queue in shared memory; full queues get the
// position at t, the field, chi and the bound above, and the few photons
// kept (a few percent) the draws and the rate, so this work is paid by full
// warps instead of by every warp that holds one such photon.  Results are
// those of testing every photon.  Optical depth updates every photon's tau
// and tests each.
// ---------------------------------------------------------------------------
template <int FORM>
__device__ __forceinline__ bool sfp_pair_possible(const sfp_run_dev* __restrict__ R, const sfp_qed_smem& T,
                                                  const float* __restrict__ pb, const sfp_segment& S,
                                                  const double* __restrict__ P, double x, double y, double z,
                                                  double ux, double uy, double uz, double t) {
    using namespace sfp;
    if (FORM == SFP_FORM_FP64) {
        double F[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (S.push) sfp_field_program(x, y, z, t, P, F);
        const double ig = inv_gamma_photon(ux, uy, uz);
        const double chi = chi_of(F, ux, uy, uz, ig);
        if (chi == 0.0 || chi < T.chi_pair_min) return false;
        return !((double)pb[sfp_pair_bin(__double2float_ru(chi))] * (R->dt * ig) < 0x1p-53);
    } else {
        // straight-line: every condition is combined at the end (no early exit)
        float F[6];
        sfp_field_program32(x, y, z, t, P, F);
        const bool field = S.push && (F[0] != 0.f || F[1] != 0.f || F[2] != 0.f || F[3] != 0.f || F[4] != 0.f ||
                                      F[5] != 0.f);
        const float g = sfp32::gamma_of(ux, uy, uz, true);
        const float chi = sfp32::chi_of(F, sfp32::d2f(ux), sfp32::d2f(uy), sfp32::d2f(uz), g);
        const bool some = chi > 0.0f && !((double)chi < T.chi_pair_min);
        return field & some & !(pb[sfp_pair_bin(chi)] * __fdividef(sfp32::d2f(R->dt), g) < 0x1p-33f);
    }
}

// chi per unit of gamma that no photon can exceed in this instance's field:
// chi <= gamma (|E| + c|B|) / E_s, with sfp_field_bound(P) >= |E| + c|B| over
// all space and time (generated with the field program), rounded up with a
// margin for the rounding of the computed chi; +inf when the field has no
// bound (a focused pulse, a user callable)
SFP_DEVICE_INLINE float sfp_chi_per_gamma(const double* __restrict__ P) {
    const double b = sfp_field_bound(P);
    if (!(b < 1e299)) return __int_as_float(0x7f800000);
    return __double2float_ru(b * (1.0 / sfp32::kEs) * (1.0 + 0x1p-10));
}

// Whether a photon's pair test can pass anywhere in the field, from its
// energy alone: its chi is at most gamma cpg, and pbmax (the prefix maximum
// of the pair-rate bound table, nondecreasing in chi) at that chi bounds the
// rate.  False implies that sfp_pair_possible is false for this photon (the
// same gamma and dt / gamma, a larger chi bin, a larger bound), so such a
// photon skips the field evaluation: results are those of testing it.
template <int FORM>
__device__ __forceinline__ bool sfp_pair_reachable(float cpg, const float* __restrict__ pbmax, double ux, double uy,
                                                   double uz, double dt) {
    using namespace sfp;
    if (FORM == SFP_FORM_FP64) {
        const double ig = inv_gamma_photon(ux, uy, uz);
        const float chimax = __double2float_ru((double)cpg / ig);
        return !((double)pbmax[sfp_pair_bin(chimax)] * (dt * ig) < 0x1p-53);
    } else {
        const float g = sfp32::gamma_of(ux, uy, uz, true);
        return !(pbmax[sfp_pair_bin(g * cpg)] * __fdividef(sfp32::d2f(dt), g) < 0x1p-33f);
    }
}

// a warp's queue of photons whose pair test can pass: tile index and, with STATE, the stored state
// (the float32 form: no second read of their rows); without it the batch
// reads the rows again (the float64 form, whose kernel has no registers to
// spare for the state held across a batch)
template <bool STATE>
struct sfp_pair_queue {
    unsigned short e[32];
};
template <>
struct sfp_pair_queue<true> {
    double x[32], y[32], z[32], ux[32], uy[32], uz[32];
    unsigned short e[32];
};

// the n queued photons (n <= 32), one per lane: their positions at t, the
// field filter (sfp_pair_possible), then the full pair test of those it
// keeps; a converted photon is marked and its delta stored; returns the
// events.  Every lane runs the filter (lanes past n on zeros, masked), as
// the field program votes across the warp.
template <int FORM, bool STATE>
__device__ __forceinline__ unsigned int sfp_pair_batch(const sfp_run_dev* __restrict__ R, const sfp_qed_smem& T,
                                                       const float* __restrict__ pb, const sfp_segment& S,
                                                       const sfp_instance& I, const double* __restrict__ P,
                                                       char* const* D, const sfp_pair_queue<STATE>& q,
                                                       unsigned int n, long long base, double t, double dt,
                                                       unsigned int step, double lag) {
    using namespace sfp;
    const int lane = threadIdx.x & 31;
    const bool in = (unsigned int)lane < n;
    const int e = in ? (int)q.e[lane] : 0;
    double x = 0.0, y = 0.0, z = 0.0, ux = 0.0, uy = 0.0, uz = 0.0;
    if (in) {
        if constexpr (STATE) {
            x = q.x[lane], y = q.y[lane], z = q.z[lane];
            ux = q.ux[lane], uy = q.uy[lane], uz = q.uz[lane];
        } else {  // the row again (indices only in the float64 form's queue)
            x = __ldcg(reinterpret_cast<const double*>(D[0]) + e), y = __ldcg(reinterpret_cast<const double*>(D[1]) + e);
            z = __ldcg(reinterpret_cast<const double*>(D[2]) + e), ux = __ldcg(reinterpret_cast<const double*>(D[3]) + e);
            uy = __ldcg(reinterpret_cast<const double*>(D[4]) + e), uz = __ldcg(reinterpret_cast<const double*>(D[5]) + e);
        }
    }
    if (S.push) photon_shift<FORM>(x, y, z, ux, uy, uz, dt, lag);  // the stored position advanced to t
    const bool keep = in & sfp_pair_possible<FORM>(R, T, pb, S, P, x, y, z, ux, uy, uz, t);
    bool ev = false;
    if (__any_sync(0xffffffffu, keep)) {
        if (keep) {
            double tau = 0.0, delta = 0.0;
            ev = sfp_pair_event<FORM, SFP_QED_REJECTION>(R, T, S, I, P, x, y, z, ux, uy, uz, t, step, base + e, tau,
                                                         delta);
            if (ev) {
                reinterpret_cast<unsigned char*>(D[6])[e] = SFP_MARK;
                reinterpret_cast<double*>(D[7])[e] = delta;
            }
        }
    }
    return __popc(__ballot_sync(0xffffffffu, ev));
}

template <bool STATE>
__device__ __forceinline__ void sfp_pair_enqueue(sfp_pair_queue<STATE>& q, unsigned int k, int e, double x, double y,
                                                 double z, double ux, double uy, double uz) {
    q.e[k] = (unsigned short)e;
    if constexpr (STATE) {
        q.x[k] = x;
        q.y[k] = y;
        q.z[k] = z;
        q.ux[k] = ux;
        q.uy[k] = uy;
        q.uz[k] = uz;
    }
}

// one tile of photons (`left` particles of its segment from its first on);
// returns its events
template <int FORM, int QED, int STAGES, bool LONG>
__device__ __forceinline__ unsigned int sfp_photon_tile(const sfp_run_dev* __restrict__ R, const sfp_qed_smem& T,
                                                        const float* s_pb, const float* s_pbmax, const sfp_segment& S,
                                                        char** desc, unsigned char* ring,
                                                        sfp_pair_queue<FORM == SFP_FORM_FP32>& q, int PT,
                                                        long long base, long long left, double t, double dt,
                                                        unsigned int step, double lag) {
    using namespace sfp;
    constexpr int OD = QED == SFP_QED_OPTICAL_DEPTH ? 1 : 0;
    constexpr bool QUEUE = QED == SFP_QED_REJECTION;
    constexpr int NC = 6 + OD;
    constexpr int SB = sfp_ring<NC>::STAGE_BYTES;
    constexpr bool QSTATE = FORM == SFP_FORM_FP32;  // the queue holds the kept photons' state
    const int lane = threadIdx.x & 31;
    char* const* D = desc;
    const sfp_instance& I = R->inst[S.instance];
    const double* __restrict__ P = sfp_field_params(I);
    const float cpg = QUEUE ? sfp_chi_per_gamma(P) : 0.0f;  // chi per gamma no photon exceeds here
            // LONG: 32 sub-steps of 32 with compile-time bounds; else sub-steps up
            // to the tile's last photon (`len`: the tile length or fewer at a
            // segment's end)
            const int len = LONG ? SFP_TILE_MAX : (int)min(left, (long long)PT);
            const bool bw = S.bw != 0, push = S.push != 0;
            __syncwarp();  // the previous tile's lanes are done with its descriptor, stages and queue
            if (lane < NC + 2) desc[lane] = sfp_desc_slot<QED, false>(S, lane, base);
            __syncwarp();
            unsigned int cnt = 0, qn = 0;
            const bool full = LONG ? left >= (long long)SFP_TILE_MAX : len == PT;
            // full long tiles of the float32 form without optical depth: each
            // lane's three component copies (components 2k + lane/16, k = 0..2)
            // read from per-tile pointers held in registers, lanes 0-1 copy the
            // flags; no descriptor reads per stage.  (The float64 form and the
            // any-tile kernel have no registers to spare for them.)
            constexpr bool REGPTR = FORM == SFP_FORM_FP32 && !OD && LONG;
            const char* q0 = nullptr;
            const char* q1 = nullptr;
            const char* q2 = nullptr;
            if (REGPTR && full) {
                const int h = lane >> 4, o = 16 * (lane & 15);
                q0 = D[h] + o;
                q1 = D[2 + h] + o;
                q2 = D[4 + h] + o;
            }
            auto issue = [&](int sb, unsigned char* dst) {
                if (REGPTR && full) {
                    const unsigned int off = (unsigned int)sb * 256u;
                    sfp::cp_async16(dst + lane * 16, q0 + off, 16u);
                    sfp::cp_async16(dst + (lane + 32) * 16, q1 + off, 16u);
                    sfp::cp_async16(dst + (lane + 64) * 16, q2 + off, 16u);
                    if (lane < 2) sfp::cp_async16(dst + (lane + 96) * 16, D[NC] + sb * 32 + 16 * lane, 16u);
                    sfp::cp_async_commit();
                } else if (full) {
                    sfp_ring_issue_full<NC, OD>(D, sb, dst, lane);
                } else {
                    sfp_ring_issue<NC, OD>(D, sb, LONG ? left : (long long)len, dst, lane);
                }
            };
    #pragma unroll
            for (int k = 0; k < STAGES - 1; ++k) {
                if (LONG || 32 * k < len) issue(k, ring + k * SB);
                else cp_async_commit();  // a short tile: nothing to fetch, the group count stays
            }
    #pragma unroll 1
            for (int sub = 0; LONG ? sub < SFP_TILE_MAX / 32 : 32 * sub < len; ++sub) {
                __syncwarp();  // every lane has read the stage about to be refilled
                const int nsub = sub + STAGES - 1;
                if (LONG ? nsub < SFP_TILE_MAX / 32 : 32 * nsub < len) issue(nsub, ring + (nsub % STAGES) * SB);
                else cp_async_commit();
                cp_async_wait<STAGES - 1>();
                __syncwarp();  // the stage of `sub` is complete for the whole warp
                const unsigned char* stg = ring + (sub % STAGES) * SB;
                const double* sd = reinterpret_cast<const double*>(stg);
                const int e = sub * 32 + lane;  // photon index from the tile's first
                const long long i = base + e;
                const bool alive = (LONG ? e < left : e < len) && stg[NC * 256 + lane] == 0;
                double x = sd[lane], y = sd[32 + lane], z = sd[64 + lane];
                double ux = sd[96 + lane], uy = sd[128 + lane], uz = sd[160 + lane];
                // the step's push is carried by the epoch (pos_epoch), so a photon
                // that does not convert stores nothing
                if (QUEUE) {
                    // from its energy alone, whether a photon's pair test can pass
                    // anywhere in the field; those that can go, with their stored
                    // state, to the queue, where the position at t, the field and
                    // the rate bound are evaluated for full warps
                    const bool keep = alive & bw & push & sfp_pair_reachable<FORM>(cpg, s_pbmax, ux, uy, uz, dt);
                    // kept photons fill the queue; a full queue is tested at once and
                    // the sub-step's remaining kept photons start the next one
                    const unsigned int kb = __ballot_sync(0xffffffffu, keep);
                    const unsigned int slot = qn + __popc(kb & ((1u << lane) - 1u)), nk = __popc(kb);
                    if (keep && slot < 32u) sfp_pair_enqueue(q, slot, e, x, y, z, ux, uy, uz);
                    if (qn + nk >= 32u) {
                        __syncwarp();  // the queue entries are written
                        cnt += sfp_pair_batch<FORM, QSTATE>(R, T, s_pb, S, I, P, D, q, 32u, base, t, dt, step, lag);
                        __syncwarp();  // every lane has read its entry
                        if (keep && slot >= 32u) sfp_pair_enqueue(q, slot - 32u, e, x, y, z, ux, uy, uz);
                        qn = qn + nk - 32u;
                    } else {
                        qn += nk;
                    }
                } else {
                    double tau = OD ? sd[192 + lane] : 0.0;
                    bool ev = false;
                    double delta = 0.0;
                    if (push) photon_shift<FORM>(x, y, z, ux, uy, uz, dt, lag);  // the position at t
                    if (alive && bw)
                        ev = sfp_pair_event<FORM, QED>(R, T, S, I, P, x, y, z, ux, uy, uz, t, step, i, tau, delta);
                    if (ev) {
                        // converted photons are pruned, not pushed (cpu.py:190); marked until their pairs are written
                        reinterpret_cast<unsigned char*>(D[NC])[e] = SFP_MARK;
                        reinterpret_cast<double*>(D[NC + 1])[e] = delta;
                    }
                    if (OD && alive && bw && D[6]) reinterpret_cast<double*>(D[6])[e] = tau;
                    cnt += __popc(__ballot_sync(0xffffffffu, ev));
                }
            }
            if (QUEUE && qn) {  // the tile's last kept photons
                __syncwarp();
                cnt += sfp_pair_batch<FORM, QSTATE>(R, T, s_pb, S, I, P, D, q, qn, base, t, dt, step, lag);
            }
    return cnt;
}

template <int FORM, int QED, int STAGES, bool LONG>
__device__ __forceinline__ void sfp_photon_body(const sfp_run_dev* __restrict__ R, int tail) {
    using namespace sfp;
    constexpr int OD = QED == SFP_QED_OPTICAL_DEPTH ? 1 : 0;
    constexpr bool QUEUE = QED == SFP_QED_REJECTION;
    constexpr int NC = 6 + OD;
    constexpr int SB = sfp_ring<NC>::STAGE_BYTES;
    extern __shared__ __align__(16) double s_tab[];
    __shared__ char* s_desc[SFP_TILE / 32][NC + 2];
    constexpr bool QSTATE = FORM == SFP_FORM_FP32;  // the queue holds the kept photons' state
    __shared__ sfp_pair_queue<QSTATE> s_q[QUEUE ? SFP_TILE / 32 : 1];  // per-warp queue of kept photons
    __shared__ float s_pb[QUEUE ? SFP_PAIR_BOUND_BINS : 1];
    __shared__ float s_pbmax[QUEUE ? SFP_PAIR_BOUND_BINS : 1];  // its prefix maximum
    sfp_step_state* st = R->st;
    if (st->skip || st->halted) return;
    if (QUEUE && st->hot_ok) return;  // sfp_hot_body runs this step
    const sfp_step_view V = sfp_view(R, st->cur);
    const long long n_tiles = V.n_ptiles;
    const unsigned int busy = sfp_busy_blocks(n_tiles, gridDim.x);
    if (blockIdx.x >= busy || n_tiles == 0) {
        sfp_tail(R, tail, s_tab);
        return;
    }
    const int PT = LONG ? SFP_TILE_MAX : V.ptile;
    const double t = V.t;
    const double dt = R->dt;
    const unsigned int step = (unsigned int)V.step;
    const double lag = V.lag;  // steps since the stored positions
    const sfp_qed_smem T = sfp_stage_tables<FORM, QED>(R, s_tab);
    if (QUEUE)
        for (int k = threadIdx.x; k < SFP_PAIR_BOUND_BINS; k += blockDim.x) {
            s_pb[k] = R->pair_bound[k];
            s_pbmax[k] = R->pair_bound[SFP_PAIR_BOUND_BINS + k];
        }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* ring = reinterpret_cast<unsigned char*>(s_tab) + R->ring_off + (size_t)warp * STAGES * SB;
    sfp_pair_queue<QSTATE>& q = s_q[QUEUE ? warp : 0];

    int tk = 0;
    if (lane == 0) tk = atomicAdd(&st->pticket, 1);
    long long tile = __shfl_sync(0xffffffffu, tk, 0);
    while (tile < n_tiles) {
        if (lane == 0) tk = atomicAdd(&st->pticket, 1);  // next ticket, in flight during this tile
        const int pos = sfp_find_group_pos(V.p_start, R->pg.n_seg, tile);
        const int si = R->pg.seg[pos];
        const long long N = V.n_buf[si];
        const long long base = (tile - V.p_start[pos]) * (long long)PT;
        if (base >= N) {  // alignment padding between segments: no photons
            if (lane == 0) R->pg.tile_cnt[tile] = 0u;
            tile = __shfl_sync(0xffffffffu, tk, 0);
            continue;
        }
        const unsigned int cnt = sfp_photon_tile<FORM, QED, STAGES, LONG>(
            R, T, s_pb, s_pbmax, R->seg[si], s_desc[warp], ring, q, PT, base, N - base, t, dt, step, lag);
        if (lane == 0) {
            R->pg.tile_cnt[tile] = cnt;
            if (cnt) atomicAdd(&R->pg.super_cnt[tile / SFP_SUPER_TILE], cnt);
        }
        tile = __shfl_sync(0xffffffffu, tk, 0);
    }
    sfp_tail(R, tail, s_tab);
}

// ---------------------------------------------------------------------------
// Hot photons (rejection sampling).  Whether a photon can create a pair
// anywhere in the field depends on its energy alone (sfp_pair_reachable), and
// a photon's energy never changes: in a cascade three photons in four are
// too soft for good.  A call of several steps therefore copies the others
// once (sfp_hot_build), appends new ones as they are born (sfp_write_photon),
// and its steps visit only that store: 40 bytes (float32 form) or 52 of each
// hot photon instead of 49 of every photon.  Nothing else changes: an entry
// holds the stored position (as of pos_epoch, which no step moves) and the
// momentum its tests read, events are marked in the segment and counted in
// its tiles, so draws, results and their order are those of the full kernel.
// The store lives for one call: buffers, flags and counts may change between
// calls.  When its room runs out, hot_ok goes to 0 and the steps run the full
// kernel; a field without a bound gets no store (sfp_hot_bounded_body).
// B200, a0 = 200, 24 % of the photons hot: 2.4e7 photons, float32 form 250 ->
// 89 us a step; 1.2e7 photons, float64 form 502 -> 172 us (113 with fewer
// divisions in sfp_device.cuh).
// ---------------------------------------------------------------------------
template <int FORM>
struct sfp_hot_real {
    using type = double;
};
template <>
struct sfp_hot_real<SFP_FORM_FP32> {
    using type = float;
};

template <int FORM>
SFP_DEVICE_INLINE void sfp_hot_put(const sfp_run_dev* __restrict__ R, long long e, unsigned int idx, double x, double y,
                                   double z, double ux, double uy, double uz) {
    using real = typename sfp_hot_real<FORM>::type;
    const sfp_hot_dev& H = R->hot;
    H.x[e] = x;
    H.y[e] = y;
    H.z[e] = z;
    if constexpr (FORM == SFP_FORM_FP64) {
        static_cast<real*>(H.ux)[e] = ux;
        static_cast<real*>(H.uy)[e] = uy;
        static_cast<real*>(H.uz)[e] = uz;
    } else {
        static_cast<real*>(H.ux)[e] = sfp32::d2f(ux);
        static_cast<real*>(H.uy)[e] = sfp32::d2f(uy);
        static_cast<real*>(H.uz)[e] = sfp32::d2f(uz);
    }
    H.idx[e] = idx;
}

// whether every field that a pair-creating photon flies in has a bound, to
// st->hot_ok (one block).  Where one has none (a focused pulse, a user callable)
// every photon is hot: the run keeps no store and takes no memory for one.
__device__ __forceinline__ void sfp_hot_bounded_body(const sfp_run_dev* __restrict__ R) {
    __shared__ int s_all;
    if (threadIdx.x == 0) s_all = 1;
    __syncthreads();
    for (int j = threadIdx.x; j < R->pg.n_seg; j += blockDim.x) {
        const sfp_segment& S = R->seg[R->pg.seg[j]];
        if (S.bw && S.push && !(sfp_chi_per_gamma(sfp_field_params(R->inst[S.instance])) < __int_as_float(0x7f800000)))
            s_all = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) R->st->hot_ok = s_all;
}

// copies the hot photons of every segment that creates pairs, a warp per
// photon tile (the plan of the call's first step); one count per tile
template <int FORM>
__device__ __forceinline__ void sfp_hot_build_body(const sfp_run_dev* __restrict__ R) {
    __shared__ unsigned short s_list[SFP_TILE / 32][SFP_TILE_MAX];
    __shared__ float s_pbmax[SFP_PAIR_BOUND_BINS];
    sfp_step_state* st = R->st;
    if (st->skip || st->halted) return;
    const sfp_step_view V = sfp_view(R, st->cur);
    for (int k = threadIdx.x; k < SFP_PAIR_BOUND_BINS; k += blockDim.x)
        s_pbmax[k] = R->pair_bound[SFP_PAIR_BOUND_BINS + k];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double dt = R->dt;
    unsigned short* list = s_list[warp];
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long tile = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile < V.n_ptiles; tile += nw) {
        const int pos = sfp_find_group_pos(V.p_start, R->pg.n_seg, tile);
        const int si = R->pg.seg[pos];
        const sfp_segment& S = R->seg[si];
        if (!S.bw || !S.push) continue;
        const long long base = (tile - V.p_start[pos]) * (long long)V.ptile;
        const int len = (int)min(V.n_buf[si] - base, (long long)V.ptile);
        const float cpg = sfp_chi_per_gamma(sfp_field_params(R->inst[S.instance]));
        if (!(cpg < __int_as_float(0x7f800000))) {  // no bound (parameters changed since the run asked)
            if (lane == 0) st->hot_ok = 0;
            return;
        }
        int n = 0;
        for (int e0 = 0; e0 < len; e0 += 32) {
            const int e = e0 + lane;
            bool keep = false;
            if (e < len && S.pruned[base + e] == 0)
                keep = sfp_pair_reachable<FORM>(cpg, s_pbmax, S.ux[base + e], S.uy[base + e], S.uz[base + e], dt);
            const unsigned int b = __ballot_sync(0xffffffffu, keep);
            if (keep) list[n + __popc(b & ((1u << lane) - 1u))] = (unsigned short)e;
            n += __popc(b);
        }
        if (n == 0) continue;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&R->hot.count[si], (unsigned long long)n);
        at = __shfl_sync(0xffffffffu, at, 0);
        if ((long long)at + n > R->hot.cap[si]) {
            if (lane == 0) st->hot_ok = 0;
            return;
        }
        __syncwarp();
        for (int k = lane; k < n; k += 32) {
            const long long i = base + list[k];
            sfp_hot_put<FORM>(R, R->hot.start[si] + (long long)at + k, (unsigned int)i, S.x[i], S.y[i], S.z[i], S.ux[i],
                              S.uy[i], S.uz[i]);
        }
        __syncwarp();
    }
}

// one hot photon's state and index
template <int FORM>
struct sfp_hot_entry {
    double x, y, z;
    typename sfp_hot_real<FORM>::type ux, uy, uz;
    unsigned int idx;
};
template <int FORM>
SFP_DEVICE_INLINE sfp_hot_entry<FORM> sfp_hot_get(const sfp_hot_dev& H, long long e, bool in) {
    using real = typename sfp_hot_real<FORM>::type;
    sfp_hot_entry<FORM> v;
    v.x = v.y = v.z = 0.0;
    v.ux = v.uy = v.uz = (real)1;
    v.idx = SFP_HOT_DEAD;
    if (in) {
        v.idx = H.idx[e];
        v.x = H.x[e];
        v.y = H.y[e];
        v.z = H.z[e];
        v.ux = static_cast<const real*>(H.ux)[e];
        v.uy = static_cast<const real*>(H.uy)[e];
        v.uz = static_cast<const real*>(H.uz)[e];
    }
    return v;
}

// hot photons that the field test keeps, waiting for their draws: chi, gamma
// (float64: 1/gamma) and where they are
template <int FORM>
struct sfp_draw_queue {
    typename sfp_hot_real<FORM>::type chi[64], g[64];
    unsigned int e[64], idx[64];
};

// the draws and the rate of up to 32 queued photons (entries q0 ..), one per lane
template <int FORM>
__device__ __forceinline__ void sfp_hot_draw(const sfp_run_dev* __restrict__ R, const sfp_qed_smem& T,
                                             const sfp_segment& S, const sfp_instance& I, const sfp_step_view& V,
                                             int pos, const sfp_draw_queue<FORM>& q, unsigned int n, long long first,
                                             unsigned int step) {
    using namespace sfp;
    const int lane = threadIdx.x & 31;
    bool ev = false;
    double d = 0.0;
    unsigned int idx = 0, e = 0;
    if ((unsigned int)lane < n) {
        idx = q.idx[lane];
        e = q.e[lane];
        if constexpr (FORM == SFP_FORM_FP64) {
            double r1, r2;
            sfp_step_uniform2(I.seed, S.stream, step, 0u, (long long)idx, r1, r2);
            ev = pair_event_rs(q.chi[lane], q.g[lane], R->dt, r1, r2, T.iAt, T.dAt, T.zN, T.zmax, d);
        } else {
            const float chi = q.chi[lane], g = q.g[lane];
            float r1, r2;
            sfp_step_uniform2f(I.seed, S.stream, step, 0u, (long long)idx, r1, r2);
            const float kRate = (float)((kAlpha * kMe) * (kC * kC) / kHbar);
            const float base = __fdividef(1.0f, (r1 * (1.0f - r1)) * chi);
            const float W = kRate * sfp32::rate_core(chi, base, T.iAf, T.dAf, T.inv_dzf, T.zN, T.base_maxf, -1.0f);
            ev = r2 < W * __fdividef(sfp32::d2f(R->dt), g);
            d = (double)r1;
        }
    }
    if (ev) {
        S.pruned[idx] = SFP_MARK;
        S.delta[idx] = d;
        R->hot.idx[first + e] = SFP_HOT_DEAD;
        const long long tile = V.p_start[pos] + (long long)(idx / (unsigned int)V.ptile);
        atomicAdd(&R->pg.tile_cnt[tile], 1u);
        atomicAdd(&R->pg.super_cnt[tile / SFP_SUPER_TILE], 1u);
    }
}

#define SFP_HOT_TILE 256
// the photon kernel over the store: per entry the position at t, the field,
// chi and the rate bound (sfp_pair_possible); those it keeps are queued and
// get their draws 32 at a time
template <int FORM>
__device__ __forceinline__ void sfp_hot_body(const sfp_run_dev* __restrict__ R, int tail) {
    using namespace sfp;
    using real = typename sfp_hot_real<FORM>::type;
    extern __shared__ __align__(16) double s_tab[];
    __shared__ sfp_draw_queue<FORM> s_q[SFP_TILE / 32];
    __shared__ float s_pb[SFP_PAIR_BOUND_BINS];
    sfp_step_state* st = R->st;
    if (st->skip || st->halted || !st->hot_ok) return;
    const sfp_step_view V = sfp_view(R, st->cur);
    const double t = V.t, dt = R->dt, lag = V.lag;
    const unsigned int step = (unsigned int)V.step;
    const sfp_qed_smem T = sfp_stage_tables<FORM, SFP_QED_REJECTION>(R, s_tab);
    for (int k = threadIdx.x; k < SFP_PAIR_BOUND_BINS; k += blockDim.x) s_pb[k] = R->pair_bound[k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the segments' first tiles, from their entries (in the room of the rings)
    long long* const first_tile = reinterpret_cast<long long*>(reinterpret_cast<unsigned char*>(s_tab) + R->ring_off);
    const int ng = R->pg.n_seg;
    if (warp == 0) {
        long long carry = 0;
        for (int j0 = 0; j0 < ng; j0 += 32) {
            const int j = j0 + lane;
            const long long own =
                j < ng ? ((long long)R->hot.count[R->pg.seg[j]] + SFP_HOT_TILE - 1) / SFP_HOT_TILE : 0;
            long long inc = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            if (j < ng) first_tile[j] = carry + inc - own;
            carry += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) first_tile[ng] = carry;
    }
    __syncthreads();
    const long long n_tiles = first_tile[ng];
    sfp_draw_queue<FORM>& q = s_q[warp];
    int tk = 0;
    if (lane == 0) tk = atomicAdd(&st->pticket, 1);
    long long tile = __shfl_sync(0xffffffffu, tk, 0);
    while (tile < n_tiles) {
        if (lane == 0) tk = atomicAdd(&st->pticket, 1);  // next ticket, in flight during this tile
        const int pos = sfp_find_group_pos(first_tile, ng, tile);
        const int si = R->pg.seg[pos];
        const sfp_segment& S = R->seg[si];
        const sfp_instance& I = R->inst[S.instance];
        const double* __restrict__ P = sfp_field_params(I);
        const long long e0 = (tile - first_tile[pos]) * (long long)SFP_HOT_TILE;
        const long long first = R->hot.start[si] + e0;  // the tile's first entry
        const int len = (int)min((long long)R->hot.count[si] - e0, (long long)SFP_HOT_TILE);
        unsigned int qn = 0;
        sfp_hot_entry<FORM> next = sfp_hot_get<FORM>(R->hot, first + lane, lane < len);
#pragma unroll 1
        for (int k0 = 0; k0 < len; k0 += 32) {
            const sfp_hot_entry<FORM> v = next;
            if (k0 + 32 < len) next = sfp_hot_get<FORM>(R->hot, first + k0 + 32 + lane, k0 + 32 + lane < len);
            // every lane runs the test, as the field program votes across the warp
            double x = v.x, y = v.y, z = v.z;
            real chi, g;
            bool keep;
            if constexpr (FORM == SFP_FORM_FP64) {
                photon_shift<FORM>(x, y, z, v.ux, v.uy, v.uz, dt, lag);
                double F[6];
                sfp_field_program(x, y, z, t, P, F);
                g = inv_gamma_photon(v.ux, v.uy, v.uz);
                chi = chi_of(F, v.ux, v.uy, v.uz, g);
                keep = !(chi == 0.0 || chi < T.chi_pair_min) &&
                       !((double)s_pb[sfp_pair_bin(__double2float_ru(chi))] * (dt * g) < 0x1p-53);
            } else {
                const float a = sfp32::d2f(kC * dt) * rsqrtf(v.ux * v.ux + v.uy * v.uy + v.uz * v.uz);
                x += lag * (double)(a * v.ux);
                y += lag * (double)(a * v.uy);
                z += lag * (double)(a * v.uz);
                float F[6];
                sfp_field_program32(x, y, z, t, P, F);
                const bool field = F[0] != 0.f || F[1] != 0.f || F[2] != 0.f || F[3] != 0.f || F[4] != 0.f || F[5] != 0.f;
                g = sqrtf(v.ux * v.ux + v.uy * v.uy + v.uz * v.uz);
                chi = sfp32::chi_of(F, v.ux, v.uy, v.uz, g);
                const bool some = chi > 0.0f && !((double)chi < T.chi_pair_min);
                keep = field & some & !(s_pb[sfp_pair_bin(chi)] * __fdividef(sfp32::d2f(dt), g) < 0x1p-33f);
            }
            keep = keep & (v.idx != SFP_HOT_DEAD);
            const unsigned int kb = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const unsigned int at = qn + __popc(kb & ((1u << lane) - 1u));
                q.chi[at] = chi;
                q.g[at] = g;
                q.e[at] = (unsigned int)(k0 + lane);
                q.idx[at] = v.idx;
            }
            qn += __popc(kb);
            if (qn >= 32u) {
                __syncwarp();  // the entries are written
                sfp_hot_draw<FORM>(R, T, S, I, V, pos, q, 32u, first, step);
                __syncwarp();  // and read
                if ((unsigned int)lane < qn - 32u) {  // the rest moves to the front
                    q.chi[lane] = q.chi[32 + lane];
                    q.g[lane] = q.g[32 + lane];
                    q.e[lane] = q.e[32 + lane];
                    q.idx[lane] = q.idx[32 + lane];
                }
                qn -= 32u;
            }
        }
        if (qn) {
            __syncwarp();
            sfp_hot_draw<FORM>(R, T, S, I, V, pos, q, qn, first, step);
        }
        __syncwarp();  // the queue is read before the next tile fills it
        tile = __shfl_sync(0xffffffffu, tk, 0);
    }
    sfp_tail(R, tail, s_tab);
}

// ---------------------------------------------------------------------------
// Appends.  The massive group's tile counters and then the photon group's
// are dealt to the warps by stride (warp w: tiles w, w + nw, ...), read 32
// at a time, one per lane; for a tile with events the warp adds the counts of
// the earlier tiles of its super-tile to the super-tile's prefix, gathers
// the tile's marked particles in index order into shared memory (16 flags
// per lane per pass) and then handles 32 of them at a time, so every lane
// works: the k-th marked particle's children go to slot
// n_buffered(start of step) + prefix + k.
//   massive: the photon (cpu.py:89-116) from the parent's state at t,
//            pushed; the parent's recoil (cpu.py:76-87) and push; unmarked;
//   photon:  e- with delta u and e+ with (1 - delta) u (cpu.py:119-189),
//            both pushed; the photon pruned.
// ---------------------------------------------------------------------------
template <int FORM>
__device__ __forceinline__ void sfp_write_pair_child(const sfp_segment& D, long long slot, const double* __restrict__ P,
                                                     double x, double y, double z, double ux, double uy, double uz,
                                                     double t, double dt) {
    using namespace sfp;
    if (D.push) {
        double sx = 0.0, sy = 0.0, sz = 0.0;
        if (FORM == SFP_FORM_FP64) push_massive(x, y, z, ux, uy, uz, sx, sy, sz, D, P, t, dt);
        else push_massive32<true>(x, y, z, ux, uy, uz, sx, sy, sz, D, P, push_consts32(D, t, dt));
    }
    D.x[slot] = x;
    D.y[slot] = y;
    D.z[slot] = z;
    D.ux[slot] = ux;
    D.uy[slot] = uy;
    D.uz[slot] = uz;
    if (D.spin) {
        D.sx[slot] = 0.0;
        D.sy[slot] = 0.0;
        D.sz[slot] = 0.0;
    }
    if (D.tau) D.tau[slot] = 0.0;
    D.pruned[slot] = 0;
}

template <int FORM>
__device__ __forceinline__ void sfp_write_photon(const sfp_run_dev* __restrict__ R, const sfp_segment& S, long long i,
                                                 long long rank, long long pre, const double* __restrict__ P,
                                                 const sfp_step_view& V, double dt, float cpg) {
    using namespace sfp;
    const double t = V.t, lag = V.lag;
    const sfp_segment& D = R->seg[S.photon_dest];
    const long long slot = V.n_buf[S.photon_dest] + pre + rank;
    double x = __ldcg(S.x + i), y = __ldcg(S.y + i), z = __ldcg(S.z + i);
    double ux = __ldcg(S.ux + i), uy = __ldcg(S.uy + i), uz = __ldcg(S.uz + i);
    const double d = __ldcg(S.delta + i);
    double cx = x, cy = y, cz = z;
    const double cux = d * ux, cuy = d * uy, cuz = d * uz;
    // the child is pushed in its creation step (simulation.py:117-121): at
    // the next step it is at x + one push, so it is stored `lag` pushes
    // behind x, as of pos_epoch like every photon of its segment
    if (D.push) photon_shift<FORM>(cx, cy, cz, cux, cuy, cuz, dt, -lag);
    D.x[slot] = cx;
    D.y[slot] = cy;
    D.z[slot] = cz;
    D.ux[slot] = cux;
    D.uy[slot] = cuy;
    D.uz[slot] = cuz;
    if (D.tau) D.tau[slot] = 0.0;
    D.pruned[slot] = 0;
    if (cpg >= 0.0f && D.bw && D.push) {  // the call keeps a store of hot photons
        const unsigned int act = __activemask();
        const bool keep = sfp_pair_reachable<FORM>(cpg, R->pair_bound + SFP_PAIR_BOUND_BINS, cux, cuy, cuz, dt);
        const unsigned int kb = __ballot_sync(act, keep);
        if (kb) {
            const int lane = threadIdx.x & 31, lead = __ffs(kb) - 1;
            unsigned long long at = 0;
            if (lane == lead) at = atomicAdd(&R->hot.count[S.photon_dest], (unsigned long long)__popc(kb));
            at = __shfl_sync(act, at, lead) + __popc(kb & ((1u << lane) - 1u));
            if (keep) {
                if ((long long)at < R->hot.cap[S.photon_dest])
                    sfp_hot_put<FORM>(R, R->hot.start[S.photon_dest] + (long long)at, (unsigned int)slot, cx, cy, cz,
                                      cux, cuy, cuz);
                else
                    R->st->hot_ok = 0;  // no room: the following steps run the full kernel
            }
        }
    }
    if (S.rr == SFP_RR_PHOTON) {
        const double f = 1.0 - d;
        // (a product of its own, not fused into the push: every kernel rounds alike)
        ux = __dmul_rn(ux, f);
        uy = __dmul_rn(uy, f);
        uz = __dmul_rn(uz, f);
    }
    if (S.push) {
        double sx = 0.0, sy = 0.0, sz = 0.0;
        if (S.spin) {
            sx = __ldcg(S.sx + i);
            sy = __ldcg(S.sy + i);
            sz = __ldcg(S.sz + i);
        }
        if (FORM == SFP_FORM_FP64) push_massive(x, y, z, ux, uy, uz, sx, sy, sz, S, P, t, dt);
        else push_massive32<true>(x, y, z, ux, uy, uz, sx, sy, sz, S, P, push_consts32(S, t, dt));
        S.x[i] = x;
        S.y[i] = y;
        S.z[i] = z;
        if (S.spin) {
            S.sx[i] = sx;
            S.sy[i] = sy;
            S.sz[i] = sz;
        }
    }
    if (S.push || S.rr == SFP_RR_PHOTON) {
        S.ux[i] = ux;
        S.uy[i] = uy;
        S.uz[i] = uz;
    }
    S.pruned[i] = 0;
}

template <int FORM>
__device__ __forceinline__ void sfp_write_pair(const sfp_run_dev* __restrict__ R, const sfp_segment& S, long long i,
                                               long long rank, long long pre, const double* __restrict__ P,
                                               const sfp_step_view& V, double dt) {
    const double t = V.t, lag = V.lag;
    const double d = __ldcg(S.delta + i);
    double px = __ldcg(S.x + i), py = __ldcg(S.y + i), pz = __ldcg(S.z + i);
    const double pux = __ldcg(S.ux + i), puy = __ldcg(S.uy + i), puz = __ldcg(S.uz + i);
    // the converted photon at t, written out: it is pruned, and pruned
    // photons keep their stored position (no later advance)
    if (S.push) {
        sfp::photon_shift<FORM>(px, py, pz, pux, puy, puz, dt, lag);
        S.x[i] = px;
        S.y[i] = py;
        S.z[i] = pz;
    }
    S.pruned[i] = 1;
    const long long be = V.n_buf[S.ele_dest] + pre + rank;
    const long long bp = V.n_buf[S.pos_dest] + pre + rank;
    sfp_write_pair_child<FORM>(R->seg[S.ele_dest], be, P, px, py, pz, __dmul_rn(d, pux), __dmul_rn(d, puy),
                               __dmul_rn(d, puz), t, dt);
    const double d2 = 1.0 - d;
    sfp_write_pair_child<FORM>(R->seg[S.pos_dest], bp, P, px, py, pz, __dmul_rn(d2, pux), __dmul_rn(d2, puy),
                               __dmul_rn(d2, puz), t, dt);
}

// (a unit of U tiles: they follow one another in a segment, so it is one
// tile of U times the length whose first tile is `tile`)
template <int FORM, bool MASSIVE>
__device__ __forceinline__ void sfp_append_tile(const sfp_run_dev* __restrict__ R, const sfp_group_dev& G,
                                                const sfp_step_view& V, long long tile, unsigned int c,
                                                unsigned short* list, double dt, bool hot, int U) {
    using namespace sfp;
    const int PT = MASSIVE ? V.mtile : V.ptile;
    const int UT = PT * U;  // the unit's particles
    const long long* start = MASSIVE ? V.m_start : V.p_start;
    const int lane = threadIdx.x & 31;
    const long long s = tile / SFP_SUPER_TILE;
    unsigned int part = 0u;
    for (long long k = s * SFP_SUPER_TILE + lane; k < tile; k += 32) part += __ldcg(&G.tile_cnt[k]);
    const long long pre = __ldcg(&G.super_pre[s]) + (long long)warp_sum(part);
    const int pos = sfp_find_group_pos(start, G.n_seg, tile);
    const sfp_segment& S = R->seg[G.seg[pos]];
    const double* __restrict__ P = sfp_field_params(R->inst[S.instance]);
    const long long N = V.n_buf[G.seg[pos]];
    const long long base = (tile - start[pos]) * (long long)PT;
    const int len = (int)min(N - base, (long long)UT);  // the unit's particles
    // chi per gamma no photon exceeds here, where new photons may enter the store of hot ones
    const float cpg = MASSIVE && hot ? sfp_chi_per_gamma(P) : -1.0f;
    // the tile's marked particles, in index order: lane q covers 16 flags per pass
    unsigned int n = 0u;
    for (int q0 = 0; q0 < len && n < c; q0 += 512) {
        const int e0 = q0 + 16 * lane;
        const unsigned char* f = S.pruned + base + e0;
        unsigned int m = 0u;
        if (e0 + 16 <= len) {
            m = marks16(__ldcg(reinterpret_cast<const uint4*>(f)));
        } else {
            for (int b = 0; b < 16; ++b)
                if (e0 + b < len && __ldcg(f + b) == SFP_MARK) m |= 1u << b;
        }
        const unsigned int k = __popc(m);
        const unsigned int inc = warp_incl_scan(k);
        unsigned int w = n + inc - k;
        while (m) {
            const int b = __ffs(m) - 1;
            m &= m - 1u;
            if (w < (unsigned int)len) list[w] = (unsigned short)(e0 + b);
            ++w;
        }
        n += __shfl_sync(0xffffffffu, inc, 31);
    }
    __syncwarp();
    // never more children than the scan counted and made room for
    n = min(min(n, c), (unsigned int)len);
    for (unsigned int j0 = 0; j0 < n; j0 += 32) {
        const unsigned int j = j0 + lane;
        if (j < n) {
            const long long i = base + list[j];
            if (MASSIVE) sfp_write_photon<FORM>(R, S, i, j, pre, P, V, dt, cpg);
            else sfp_write_pair<FORM>(R, S, i, j, pre, P, V, dt);
        }
    }
    __syncwarp();  // the list is read before the next tile rewrites it
}

// the step of view V: children of every unit dealt to warp gw of nw
template <int FORM>
__device__ __forceinline__ void sfp_append_units(const sfp_run_dev* __restrict__ R, const sfp_step_view& V,
                                                 unsigned short* list, long long gw, long long nw, double dt,
                                                 bool hot) {
    const int lane = threadIdx.x & 31;
    const long long nm = R->any_rad ? V.n_mtiles : 0, np = R->any_bw ? V.n_ptiles : 0;
    // a unit of the massive group: as many tiles as leave one unit or more for
    // every warp, SFP_TILE_MAX particles at most
    int U = 1;
    while (nm / U > nw && V.mtile * U * 2 <= SFP_TILE_MAX && U < SFP_SUPER_TILE) U <<= 1;
    const long long um = (nm + U - 1) / U, units = um + np;
    // warp gw owns units gw, gw + nw, gw + 2 nw, ...: those with events
    // (every massive one in a cascade, a few photon tiles) spread over all
    // warps instead of queueing behind one warp per 32 neighbours
    for (long long j0 = 0; gw + j0 * nw < units; j0 += 32) {
        const long long mine = gw + (j0 + lane) * nw;
        unsigned int mc = 0u;
        if (mine < um) {
            const long long t0 = mine * U, t1 = min(nm, t0 + U);
            for (long long k = t0; k < t1; ++k) mc += __ldcg(&R->mg.tile_cnt[k]);
        } else if (mine < units) {
            mc = __ldcg(&R->pg.tile_cnt[mine - um]);
        }
        unsigned int busy = __ballot_sync(0xffffffffu, mc != 0u);
        while (busy) {
            const int b = __ffs(busy) - 1;
            busy &= busy - 1u;
            const long long tg = gw + (j0 + b) * nw;
            const unsigned int c = __shfl_sync(0xffffffffu, mc, b);
            if (tg < um) sfp_append_tile<FORM, true>(R, R->mg, V, tg * U, c, list, dt, hot, U);
            else sfp_append_tile<FORM, false>(R, R->pg, V, tg - um, c, list, dt, hot, 1);
        }
    }
}

template <int FORM>
__device__ __forceinline__ void sfp_appends_body(const sfp_run_dev* __restrict__ R) {
    __shared__ unsigned short s_list[SFP_TILE / 32][SFP_TILE_MAX];
    const sfp_step_state* st = R->st;
    if (st->skip || st->halted) return;
    const sfp_step_view V = sfp_view(R, st->cur ^ 1);  // the step whose events were scanned
    const long long n_all = (R->any_rad ? V.n_mtiles : 0) + (R->any_bw ? V.n_ptiles : 0);
    const unsigned int busy_blocks = sfp_busy_blocks(n_all, gridDim.x);
    if (blockIdx.x >= busy_blocks) return;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)busy_blocks * blockDim.x) >> 5;
    sfp_append_units<FORM>(R, V, s_list[threadIdx.x >> 5], gw, nw, R->dt, st->hot_ok != 0);
}

// ---------------------------------------------------------------------------
// Small populations: several steps in one launch (a cooperative one, every
// block resident).  A step of 1e4 e- spent 53 us in three launches of which
// no block had more than a few tiles: launch gaps (2 us each), tables staged
// anew (2-4 us each), and the rest one tile's chain of dependent operations.
// Here the tables are staged once, and a step is: every warp's tiles of both
// groups; a grid barrier (2 us); the event scan in block 0; a barrier; the
// children, while block 0 plans the next step; a barrier.  Particles, flags
// and counts that other blocks write are read past L1 (cp.async.cg, __ldcg).
// A barrier gives up after SFP_BARRIER_NS: the step's error is set and every
// block returns.  Step times against three launches, float64 / float32 form:
// 1e3 e- 49 -> 31 / 34 -> 22 us, 1e4 63 -> 40 / 41 -> 23, 1e5 151 -> 95 /
// 73 -> 37.
// ---------------------------------------------------------------------------
// A wait lies within one step, under 0.8 ms at the largest populations that this
// kernel serves: the limit is 2500 times that.
#define SFP_BARRIER_NS 2000000000ull
// segments of a run that may take this kernel
#define SFP_SMALL_SEGS 64

__device__ __forceinline__ unsigned long long sfp_clock_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// all blocks of the launch; `round` counts the barriers of the launch from 1.
// False (in every thread of the block) once the wait has run out.
__device__ __forceinline__ bool sfp_grid_barrier(sfp_step_state* st, unsigned int round) {
    __shared__ int s_in;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int want = round * gridDim.x;
        __threadfence();
        atomicAdd(&st->barrier, 1u);
        int in = 1;
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&st->barrier) : "memory");
        if (v < want) {
            const unsigned long long t0 = sfp_clock_ns();
            for (unsigned int k = 1; v < want; ++k) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&st->barrier) : "memory");
                if ((k & 255u) == 0u && v < want && sfp_clock_ns() - t0 > SFP_BARRIER_NS) {
                    in = 0;
                    break;
                }
            }
        }
        if (!in) st->error = SFP_DEV_BARRIER;
        __threadfence();
        s_in = in;
    }
    __syncthreads();
    return s_in != 0;
}

// the massive group's tile as a function of its own: compiled by itself, it
// rounds as it does in the group kernels
template <int FORM, int QED, bool SPIN>
__device__ __noinline__ unsigned int sfp_massive_tile_call(const sfp_run_dev* __restrict__ R, const sfp_qed_smem& T,
                                                           const sfp_mlp::Smem& M, const sfp_segment& S, char** desc,
                                                           unsigned char* ring, int SB, int PT, long long base,
                                                           long long left, double t, double dt, unsigned int step) {
    return sfp_massive_tile<FORM, QED, 2, SPIN, false>(R, T, M, S, desc, ring, SB, PT, base, left, t, dt, step);
}

template <int FORM, int QED>
__device__ __forceinline__ void sfp_steps_body(const sfp_run_dev* __restrict__ R, int nsteps, int end) {
    using namespace sfp;
    if (nsteps < 0) {  // a test of the barrier's time limit: the last block never arrives
        if (blockIdx.x == gridDim.x - 1) return;
        nsteps = -nsteps;
    }
    constexpr int OD = QED == SFP_QED_OPTICAL_DEPTH ? 1 : 0;
    constexpr bool QUEUE = QED == SFP_QED_REJECTION;
    constexpr int NW = SFP_TILE / 32;
    extern __shared__ __align__(16) double s_tab[];
    __shared__ char* s_desc[NW][6 + OD + 3 + 2];
    __shared__ sfp_pair_queue<FORM == SFP_FORM_FP32> s_q[QUEUE ? NW : 1];
    __shared__ float s_pb[QUEUE ? SFP_PAIR_BOUND_BINS : 1];
    __shared__ float s_pbmax[QUEUE ? SFP_PAIR_BOUND_BINS : 1];
    __shared__ long long s_start[2][SFP_SMALL_SEGS + 1], s_nbuf[SFP_SMALL_SEGS];
    __shared__ sfp_step_plan s_plan;
    __shared__ int s_cur, s_stop;
    sfp_step_state* st = R->st;
    const double dt = R->dt;
    const sfp_qed_smem T = sfp_stage_tables<FORM, QED>(R, s_tab);
    sfp_mlp::Smem& M = *reinterpret_cast<sfp_mlp::Smem*>(reinterpret_cast<unsigned char*>(s_tab) + R->mlp_off);
    if (OD && R->mlp_params) sfp_mlp::stage(M, R->mlp_params);
    if (QUEUE)
        for (int k = threadIdx.x; k < SFP_PAIR_BOUND_BINS; k += blockDim.x) {
            s_pb[k] = R->pair_bound[k];
            s_pbmax[k] = R->pair_bound[SFP_PAIR_BOUND_BINS + k];
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* const ring = reinterpret_cast<unsigned char*>(s_tab) + R->m_ring_off + (size_t)warp * R->small_ring;
    sfp_end_smem& Q = *reinterpret_cast<sfp_end_smem*>(reinterpret_cast<unsigned char*>(s_tab) + R->small_end_off);
    const long long gw = (long long)warp * gridDim.x + blockIdx.x, nw = (long long)NW * gridDim.x;
    unsigned int round = 0;
    for (int k = 0; k < nsteps; ++k) {
        // the step's plan, written by block 0 (or by the launch before)
        if (threadIdx.x == 0) {
            s_stop = __ldcg(&st->skip) | __ldcg(&st->halted) | __ldcg(&st->error);
            s_cur = __ldcg(&st->cur);
        }
        __syncthreads();
        if (s_stop) return;
        const int cur = s_cur;
        if (threadIdx.x == 0) {
            const sfp_step_plan& p = st->plan[cur];
            s_plan.t = __ldcg(&p.t);
            s_plan.step = __ldcg(&p.step);
            s_plan.n_mtiles = __ldcg(&p.n_mtiles);
            s_plan.n_ptiles = __ldcg(&p.n_ptiles);
            s_plan.mtile = __ldcg(&p.mtile);
            s_plan.ptile = __ldcg(&p.ptile);
        }
        for (int j = threadIdx.x; j < R->mg.n_seg; j += blockDim.x)
            s_start[0][j] = __ldcg(R->mg.tile_start + cur * (R->mg.n_seg + 1) + j);
        for (int j = threadIdx.x; j < R->pg.n_seg; j += blockDim.x)
            s_start[1][j] = __ldcg(R->pg.tile_start + cur * (R->pg.n_seg + 1) + j);
        for (int j = threadIdx.x; j < R->n_seg; j += blockDim.x) s_nbuf[j] = __ldcg(R->n_buf_step + cur * R->n_seg + j);
        __syncthreads();
        sfp_step_view V;
        V.t = s_plan.t;
        V.step = s_plan.step;
        V.lag = (double)(s_plan.step - st->pos_epoch);
        V.n_mtiles = s_plan.n_mtiles;
        V.n_ptiles = s_plan.n_ptiles;
        V.mtile = s_plan.mtile;
        V.ptile = s_plan.ptile;
        V.m_start = s_start[0];
        V.p_start = s_start[1];
        V.n_buf = s_nbuf;
        for (long long w = gw; w < V.n_mtiles + V.n_ptiles; w += nw) {
            const bool massive = w < V.n_mtiles;
            const sfp_group_dev& G = massive ? R->mg : R->pg;
            const long long tile = massive ? w : w - V.n_mtiles;
            const long long* start = massive ? V.m_start : V.p_start;
            const int pos = sfp_find_group_pos(start, G.n_seg, tile);
            const int si = G.seg[pos];
            const sfp_segment& S = R->seg[si];
            const int PT = massive ? V.mtile : V.ptile;
            const long long base = (tile - start[pos]) * (long long)PT;
            const long long left = V.n_buf[si] - base;
            unsigned int cnt = 0;
            if (left > 0) {  // else: alignment padding between segments
                if (!massive)
                    cnt = sfp_photon_tile<FORM, QED, 3, false>(R, T, s_pb, s_pbmax, S, s_desc[warp], ring,
                                                               s_q[QUEUE ? warp : 0], PT, base, left, V.t, dt,
                                                               (unsigned int)V.step, V.lag);
                else if (S.spin)
                    cnt = sfp_massive_tile_call<FORM, QED, true>(R, T, M, S, s_desc[warp], ring, R->m_stage_bytes,
                                                                      PT, base, left, V.t, dt, (unsigned int)V.step);
                else
                    cnt = sfp_massive_tile_call<FORM, QED, false>(R, T, M, S, s_desc[warp], ring, R->m_stage_bytes,
                                                                       PT, base, left, V.t, dt, (unsigned int)V.step);
            }
            if (lane == 0) {
                G.tile_cnt[tile] = cnt;
                if (cnt) atomicAdd(&G.super_cnt[tile / SFP_SUPER_TILE], cnt);
            }
        }
        if (!sfp_grid_barrier(st, ++round)) return;
        if (blockIdx.x == 0) sfp_end_scan(R, end, Q);
        if (!sfp_grid_barrier(st, ++round)) return;
        if (threadIdx.x == 0) s_stop = __ldcg(&st->halted);
        __syncthreads();
        if (s_stop) return;  // no room: the host resumes the step
        // the children, while block 0 plans the next step
        if (blockIdx.x == 0)
            sfp_end_plan(R, end, Q, (int)nw);
        else
            sfp_append_units<FORM>(R, V, reinterpret_cast<unsigned short*>(ring), (long long)warp * (gridDim.x - 1) + blockIdx.x - 1,
                                   (long long)NW * (gridDim.x - 1), dt, false);
        if (!sfp_grid_barrier(st, ++round)) return;
    }
}

// kernels: sfp_massive_<form>_<qed>_s<stages>_b<blocks>,
// sfp_photon_<form>_<qed>_s<stages>_b<blocks>, sfp_book_kernel, sfp_appends_<form>
// (long-tile kernels) and sfp_massive_<form>_<qed>_s<stages>_b<blocks>_t,
// sfp_photon_..._t (any tile length: the steps of small populations)
#define SFP_MASSIVE_KERNEL(FORM_S, QED_S, FORM, QED, STAGES, MINB)                                             \
    extern "C" __global__ void __launch_bounds__(SFP_TILE, MINB)                                              \
        sfp_massive_##FORM_S##_##QED_S##_s##STAGES##_b##MINB(const sfp_run_dev* __restrict__ R, int tail) {   \
        sfp_massive_body<FORM, QED, STAGES, true>(R, tail);                                                        \
    }
#define SFP_PHOTON_KERNEL(FORM_S, QED_S, FORM, QED, STAGES, MINB)                                              \
    extern "C" __global__ void __launch_bounds__(SFP_TILE, MINB)                                              \
        sfp_photon_##FORM_S##_##QED_S##_s##STAGES##_b##MINB(const sfp_run_dev* __restrict__ R, int tail) {              \
        sfp_photon_body<FORM, QED, STAGES, true>(R, tail);                                                         \
    }
#define SFP_MASSIVE_KERNEL_T(FORM_S, QED_S, FORM, QED, STAGES, MINB)                                           \
    extern "C" __global__ void __launch_bounds__(SFP_TILE, MINB)                                              \
        sfp_massive_##FORM_S##_##QED_S##_s##STAGES##_b##MINB##_t(const sfp_run_dev* __restrict__ R, int tail) {         \
        sfp_massive_body<FORM, QED, STAGES, false>(R, tail);                                                       \
    }
#define SFP_PHOTON_KERNEL_T(FORM_S, QED_S, FORM, QED, STAGES, MINB)                                            \
    extern "C" __global__ void __launch_bounds__(SFP_TILE, MINB)                                              \
        sfp_photon_##FORM_S##_##QED_S##_s##STAGES##_b##MINB##_t(const sfp_run_dev* __restrict__ R, int tail) {          \
        sfp_photon_body<FORM, QED, STAGES, false>(R, tail);                                                        \
    }

// ---------------------------------------------------------------------------
// Photon positions written out (sfp_run_sync_positions): every photon of a
// pushed photon segment that is not pruned (alive, or marked inside a step
// that stopped for room) advances by the steps since pos_epoch; pruned
// photons keep the position they were pruned at.  sfp_epoch_kernel, launched
// after it, then moves pos_epoch to the current step (a second launch, so
// that every block of the first has read the old epoch).
// ---------------------------------------------------------------------------
template <int FORM>
__device__ __forceinline__ void sfp_sync_positions_body(const sfp_run_dev* __restrict__ R) {
    const sfp_step_state* st = R->st;
    const double lag = (double)(st->step - st->pos_epoch);
    if (lag == 0.0) return;
    const double dt = R->dt;
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (int k = 0; k < R->pg.n_seg; ++k) {
        const int si = R->pg.seg[k];
        const sfp_segment& S = R->seg[si];
        if (!S.push) continue;
        const long long N = R->n_buffered[si];
        for (long long i = first; i < N; i += stride) {
            if (S.pruned[i] == 1) continue;
            double x = S.x[i], y = S.y[i], z = S.z[i];
            sfp::photon_shift<FORM>(x, y, z, S.ux[i], S.uy[i], S.uz[i], dt, lag);
            S.x[i] = x;
            S.y[i] = y;
            S.z[i] = z;
        }
    }
}

#if defined(SFP_STEP_QED_RS)
extern "C" __global__ void __launch_bounds__(256) sfp_hot_bounded_kernel(const sfp_run_dev* __restrict__ R) {
    sfp_hot_bounded_body(R);
}
#endif

extern "C" __global__ void __launch_bounds__(32) sfp_epoch_kernel(const sfp_run_dev* __restrict__ R) {
    if (threadIdx.x == 0) R->st->pos_epoch = R->st->step;
}

#if defined(SFP_STEP_FORM_FP64)
extern "C" __global__ void __launch_bounds__(SFP_TILE, 2) sfp_appends_fp64(const sfp_run_dev* __restrict__ R) {
    sfp_appends_body<SFP_FORM_FP64>(R);
}
#if defined(SFP_STEP_QED_RS)
extern "C" __global__ void __launch_bounds__(SFP_TILE, 2) sfp_steps_fp64_rs(const sfp_run_dev* __restrict__ R, int nsteps, int end) {
    sfp_steps_body<SFP_FORM_FP64, SFP_QED_REJECTION>(R, nsteps, end);
}
#else
extern "C" __global__ void __launch_bounds__(SFP_TILE, 2) sfp_steps_fp64_od(const sfp_run_dev* __restrict__ R, int nsteps, int end) {
    sfp_steps_body<SFP_FORM_FP64, SFP_QED_OPTICAL_DEPTH>(R, nsteps, end);
}
#endif
extern "C" __global__ void __launch_bounds__(256) sfp_sync_positions_fp64(const sfp_run_dev* __restrict__ R) {
    sfp_sync_positions_body<SFP_FORM_FP64>(R);
}
#if defined(SFP_STEP_QED_RS)
extern "C" __global__ void __launch_bounds__(SFP_TILE, 2) sfp_hot_fp64(const sfp_run_dev* __restrict__ R, int tail) {
    sfp_hot_body<SFP_FORM_FP64>(R, tail);
}
extern "C" __global__ void __launch_bounds__(SFP_TILE) sfp_hot_build_fp64(const sfp_run_dev* __restrict__ R) {
    sfp_hot_build_body<SFP_FORM_FP64>(R);
}
SFP_MASSIVE_KERNEL(fp64, rs, SFP_FORM_FP64, SFP_QED_REJECTION, 2, 2)
SFP_MASSIVE_KERNEL(fp64, rs, SFP_FORM_FP64, SFP_QED_REJECTION, 3, 2)
SFP_PHOTON_KERNEL(fp64, rs, SFP_FORM_FP64, SFP_QED_REJECTION, 2, 3)
SFP_PHOTON_KERNEL(fp64, rs, SFP_FORM_FP64, SFP_QED_REJECTION, 3, 3)
SFP_PHOTON_KERNEL(fp64, rs, SFP_FORM_FP64, SFP_QED_REJECTION, 3, 2)
SFP_MASSIVE_KERNEL_T(fp64, rs, SFP_FORM_FP64, SFP_QED_REJECTION, 2, 2)
SFP_PHOTON_KERNEL_T(fp64, rs, SFP_FORM_FP64, SFP_QED_REJECTION, 3, 3)
#else
SFP_MASSIVE_KERNEL(fp64, od, SFP_FORM_FP64, SFP_QED_OPTICAL_DEPTH, 2, 2)
SFP_MASSIVE_KERNEL(fp64, od, SFP_FORM_FP64, SFP_QED_OPTICAL_DEPTH, 3, 2)
SFP_PHOTON_KERNEL(fp64, od, SFP_FORM_FP64, SFP_QED_OPTICAL_DEPTH, 2, 3)
SFP_PHOTON_KERNEL(fp64, od, SFP_FORM_FP64, SFP_QED_OPTICAL_DEPTH, 3, 3)
SFP_MASSIVE_KERNEL_T(fp64, od, SFP_FORM_FP64, SFP_QED_OPTICAL_DEPTH, 2, 2)
SFP_PHOTON_KERNEL_T(fp64, od, SFP_FORM_FP64, SFP_QED_OPTICAL_DEPTH, 3, 3)
#endif
#endif
#if defined(SFP_STEP_FORM_FP32)
extern "C" __global__ void __launch_bounds__(SFP_TILE, 3) sfp_appends_fp32(const sfp_run_dev* __restrict__ R) {
    sfp_appends_body<SFP_FORM_FP32>(R);
}
#if defined(SFP_STEP_QED_RS)
extern "C" __global__ void __launch_bounds__(SFP_TILE, 2) sfp_steps_fp32_rs(const sfp_run_dev* __restrict__ R, int nsteps, int end) {
    sfp_steps_body<SFP_FORM_FP32, SFP_QED_REJECTION>(R, nsteps, end);
}
#else
extern "C" __global__ void __launch_bounds__(SFP_TILE, 2) sfp_steps_fp32_od(const sfp_run_dev* __restrict__ R, int nsteps, int end) {
    sfp_steps_body<SFP_FORM_FP32, SFP_QED_OPTICAL_DEPTH>(R, nsteps, end);
}
#endif
extern "C" __global__ void __launch_bounds__(256) sfp_sync_positions_fp32(const sfp_run_dev* __restrict__ R) {
    sfp_sync_positions_body<SFP_FORM_FP32>(R);
}
#if defined(SFP_STEP_QED_RS)
extern "C" __global__ void __launch_bounds__(SFP_TILE, 3) sfp_hot_fp32(const sfp_run_dev* __restrict__ R, int tail) {
    sfp_hot_body<SFP_FORM_FP32>(R, tail);
}
extern "C" __global__ void __launch_bounds__(SFP_TILE) sfp_hot_build_fp32(const sfp_run_dev* __restrict__ R) {
    sfp_hot_build_body<SFP_FORM_FP32>(R);
}
SFP_MASSIVE_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 2, 3)
SFP_MASSIVE_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 3, 3)
SFP_MASSIVE_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 3, 2)
SFP_MASSIVE_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 4, 2)
SFP_MASSIVE_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 2, 4)
SFP_PHOTON_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 2, 4)
SFP_PHOTON_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 3, 4)
SFP_PHOTON_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 3, 3)
SFP_PHOTON_KERNEL(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 4, 3)
SFP_MASSIVE_KERNEL_T(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 2, 3)
SFP_PHOTON_KERNEL_T(fp32, rs, SFP_FORM_FP32, SFP_QED_REJECTION, 3, 3)
#else
SFP_MASSIVE_KERNEL(fp32, od, SFP_FORM_FP32, SFP_QED_OPTICAL_DEPTH, 2, 3)
SFP_MASSIVE_KERNEL(fp32, od, SFP_FORM_FP32, SFP_QED_OPTICAL_DEPTH, 3, 2)
SFP_PHOTON_KERNEL(fp32, od, SFP_FORM_FP32, SFP_QED_OPTICAL_DEPTH, 3, 4)
SFP_PHOTON_KERNEL(fp32, od, SFP_FORM_FP32, SFP_QED_OPTICAL_DEPTH, 3, 3)
SFP_MASSIVE_KERNEL_T(fp32, od, SFP_FORM_FP32, SFP_QED_OPTICAL_DEPTH, 2, 3)
SFP_PHOTON_KERNEL_T(fp32, od, SFP_FORM_FP32, SFP_QED_OPTICAL_DEPTH, 3, 3)
#endif
#endif
#endif  // SFP_WANT_STEP

#if defined(SFP_WANT_FIELD_EVAL)

// Field evaluation of the program at particle positions (Fields.field_func,
// fields.py:31-46): the per-op boundary kernel of the NVRTC module.
extern "C" __global__ void __launch_bounds__(256)
    sfp_field_eval_kernel(const double* __restrict__ P, const double* __restrict__ x, const double* __restrict__ y,
                          const double* __restrict__ z, double t, long long N, const unsigned char* __restrict__ pruned,
                          double* __restrict__ Ex, double* __restrict__ Ey, double* __restrict__ Ez,
                          double* __restrict__ Bx, double* __restrict__ By, double* __restrict__ Bz) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
        if (pruned[i]) continue;
        double F[6];
        sfp_field_program(x[i], y[i], z[i], t, P, F);
        Ex[i] = F[0]; Ey[i] = F[1]; Ez[i] = F[2];
        Bx[i] = F[3]; By[i] = F[4]; Bz[i] = F[5];
    }
}
#endif  // SFP_WANT_FIELD_EVAL
