// Fused RKDG stage kernel for sm_100a.
//
// One CTA owns one tile of TILE consecutive elements (device order = Morton order of centroids).
// Per RK stage it does, thread = element:
//   1. loads the element's modes and writes the traces of its three faces at the edge Gauss points to shared
//      memory. Neighbours in other tiles ("halo" faces) get their face traces written by the same routine
//      from global memory, and a boundary face's ghost state (BC::Land / Tide / Flow / Function,
//      rkdg_swe_bc_land.hpp:41-66, rkdg_swe_bc_function.hpp:27-60) goes to a trace slot of its own, so that the
//      face loop below has no boundary branches. Then the thread arrives on the barrier between the traces and the
//      faces (the only other one follows the CTA's set-up, before any trace);
//   2. accumulates the volume and source integrals in registers (Problem::volume_kernel + source_kernel,
//      rkdg_swe_proc_volume.hpp:9-35, rkdg_swe_proc_source.hpp:9-18) while the other warps' traces arrive;
//   3. waits on the barrier and takes the numerical flux of its own three faces (LLF + the wet/dry fix-ups of
//      ISP::Internal, rkdg_swe_is_internal.hpp:26-95) straight into the lift. Both elements of an interface
//      evaluate the flux, each with the outward normal and the weight of its own geometry. For one shared normal the
//      formula's two values are exact negatives, as the reference's are; here they cancel to the rounding of J^-1,
//      2e-7 of the flux in FP32, and a mass flux that is itself rounding may be refused by a dry side and given by
//      the wet one. Mass of a closed basin after 4,000 steps: 6e-11 off in FP32, 4e-15 in FP64;
//   4. applies M^-1 and the SSP-RK stage combination (element.hpp:502-505,
//      explicit_ssp_rk_stepper.hpp:67-80), the wetting/drying kernel (swe_post_wet_dry.hpp:6-145, its depth
//      tests in FP64 in every precision) and the NaN scrutiny; writes the next stage state.
// What bounds it: latency and instruction issue, not bytes (15 to 46 % of the HBM rate), so it is arranged for few
// instructions and few waits. Evaluating each flux twice costs about four more LLF evaluations per element than
// one per edge of the tile, and saves the flux's way through shared memory, the edge lists, a second barrier and the
// half-empty second round of edges. Against one flux per edge between two barriers, and with the step time formed once
// per step: 524,288 triangles, p = 2, FP32, second stage: warp instructions 46.7 M -> 35.4 M, barrier stalls 1.3 -> 0.1
// per issue, cold 97.7 -> 73.6 us; 8 steps 2.43 -> 1.89 ms (FP64 4.81 -> 3.70 ms); tidal channel p = 1 of 433,394 FP32
// 0.84 -> 0.54 ms; ensemble of 24 wet/dry members FP32 1.95 -> 1.30 ms.
// The master tables are compile-time constants (tables_gen.h): in the unrolled loops every table entry is an immediate and
// zero entries are skipped; the rolled ones read them from constant memory (stage_tab).
// HBM layout: component-major SoA, q[(var*ND + dof) * ne_pad + element].
#ifndef DGSW_STAGE_KERNEL_CUH
#define DGSW_STAGE_KERNEL_CUH

#include <cstdint>
#include <type_traits>

#include "../../include/dgsw_rkdg.h"
#include "function_sets.h"
#include "rk_tables.h"
#include "tables_gen.h"

namespace dgsw {

// compile-time loops
template <int N>
struct IC {
    static constexpr int value = N;
    __device__ constexpr operator int() const { return N; }
};
template <int B, int E, typename F>
__device__ __forceinline__ void sfor(F&& f) {
    if constexpr (B < E) {
        f(IC<B>{});
        sfor<B + 1, E>(f);
    }
}

// explicitly rounded operations: the two sides of an interface evaluate the flux from either side, and the
// compiler's choice of contractions must not differ between the own and the neighbour term
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// Two values of one kind, (qx, qy) or (ze, b). PK: one packed FP32 instruction of sm_100 for both
// (FFMA2 / FMUL2 / FADD2, each lane an IEEE operation); otherwise two scalar ones. The pairs are those that a
// trace vector holds side by side, so that no register moves are needed to form them.
template <typename Real>
struct Two {
    Real x, y;
};
template <bool PK, typename Real>
__device__ __forceinline__ Two<Real> fma2(Two<Real> a, Two<Real> b, Two<Real> c) {
    if constexpr (PK) {
        const float2 r = __ffma2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y), make_float2(c.x, c.y));
        return {r.x, r.y};
    } else {
        return {fma_rn(a.x, b.x, c.x), fma_rn(a.y, b.y, c.y)};
    }
}
template <bool PK, typename Real>
__device__ __forceinline__ Two<Real> fma2(Two<Real> a, Real b, Two<Real> c) {
    return fma2<PK, Real>(a, Two<Real>{b, b}, c);
}
template <bool PK, typename Real>
__device__ __forceinline__ Two<Real> mul2(Two<Real> a, Two<Real> b) {
    if constexpr (PK) {
        const float2 r = __fmul2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
        return {r.x, r.y};
    } else {
        return {mul_rn(a.x, b.x), mul_rn(a.y, b.y)};
    }
}
template <bool PK, typename Real>
__device__ __forceinline__ Two<Real> mul2(Two<Real> a, Real b) {
    return mul2<PK, Real>(a, Two<Real>{b, b});
}
template <bool PK, typename Real>
__device__ __forceinline__ Two<Real> add2(Two<Real> a, Two<Real> b) {
    if constexpr (PK) {
        const float2 r = __fadd2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
        return {r.x, r.y};
    } else {
        return {add_rn(a.x, b.x), add_rn(a.y, b.y)};
    }
}

// whether a table entry counts: the quadrature points are rounded, so entries that are zero in exact
// arithmetic come out as a few 1e-16 of the table's entries near 1
constexpr bool counts(double c) { return c > 1e-13 || c < -1e-13; }

// NaN scrutiny (scrutinize_solution after every stage, rkdg_swe_proc_serial_step.hpp:59-65): the reference
// stops at the first stage whose state holds a NaN and reports the first element (ascending ID) there.
// nan_key = (stage counter << 32) | reference element index, stage counter = step * stages + stage, kept
// as the minimum over all stages and elements of a batch: the first bad stage, then its smallest element.
struct DevStatus {
    unsigned long long nan_key;  // ~0 while no NaN has been seen
    unsigned int nan_flag;
    unsigned int wait_failed;  // a thread gave up waiting at its CTA's barrier
};

constexpr int SINE_NCONST = 10;

// What a stage needs of its time (t + dt drk[s]): the function set's time factors
struct StageTime {
    dgsw_fn_time ft;
    double sine[SINE_NCONST];  // the manufactured sine set's constants (SineSrc), in both precisions
    float sine_f[SINE_NCONST];
};

struct DevClock {
    double t;  // time at the start of the current step (ESSPRKStepper::t)
    long long step;
    StageTime at[DGSW_RK_MAX_STAGES];  // per stage of the current step
};

constexpr int FORCE_STRIDE_DEV = 9;

// Everything that depends on time alone, formed once per step for the next one: the clock itself, each
// stage's time factors (FP64 sines and cosines) and the tide / flow values at the forced faces' Gauss points.
// There are two copies, keyed by the step's parity: a step reads one while extra CTAs of its last stage's
// launch write the other, so neither a launch of its own nor the stage's CTAs wait for that arithmetic.
// Stages with the same offset drk share one set of forcing values (all of them in the reference's tables).
struct TimeArgs {
    double dt;
    double off[DGSW_RK_MAX_STAGES];  // dt drk[s]
    int nstages;
    int fn_set;
    double fn_params[16];
    int ramp_on;           // ramp_duration not almost zero
    double ramp_duration;  // days
    // tide / flow boundary forcing: per forced face its first constituent entry and count; per entry
    // frequency, forcing factor, equilibrium argument, amplitude[3] and phase[3] at the Gauss points
    const int2* fface;
    const double* fcon;
    int n_forced, ng;
    int nsets;                          // forcing value sets
    int set_stage[DGSW_RK_MAX_STAGES];  // the first stage of each set
    const DevClock* cur;                // advance from this copy (null: write `t0`, `step0` as they are)
    double t0;
    long long step0;
    DevClock* next;
    double* fval;  // [nsets][n_forced][ng] written for `next`
};

// The manufactured sine set at one stage time: ze = c1 P, qx = -c2 Q, qy = c2 R, zex = c3 Q, zey = -c3 R,
// zet = -c4 P, qxx = qyy = c5 P, qxy = qyx = c5 S, qxt = -c6 Q, qyt = c6 R with P = sx cy, Q = cx cy, R = sx sy,
// S = cx sy; c0 = 2 c5 - c4 is the continuity source's. {k, c1, c2, c3, c5, c6, c0, g, H, k / pi}
__device__ __forceinline__ void sine_constants(const double* P, StageTime& S) {
    const double k = 2.0 * M_PI / P[0], A = P[1], w = S.ft.s[2], B = P[1] * S.ft.s[2] / (2.0 * k);
    const double st = S.ft.s[0], ct = S.ft.s[1];
    const double c[SINE_NCONST] = {k,      A * ct, B * st, A * k * ct, B * k * st, B * w * ct, 2.0 * B * k * st - A * w * st,
                                   P[4],   P[2],   2.0 / P[0]};
#pragma unroll
    for (int i = 0; i < SINE_NCONST; ++i) {
        S.sine[i] = c[i];
        S.sine_f[i] = (float)c[i];
    }
}

// the ramp of ESSPRKStepper::operator++, explicit_ssp_rk_stepper.hpp:49-65 (1 without a ramp)
__device__ __forceinline__ double forcing_ramp(const TimeArgs& T, double t) {
    return T.ramp_on ? tanh(2.0 * (t / 86400.0) / T.ramp_duration) : 1.0;
}

// block 0: the clock and the stages' time factors; the others: one forcing value per thread,
// sum_con ramp * forcing_fact * amplitude_gp * cos(frequency * t + (equilib_arg - phase_gp) * PI / 180)
// with the reference's PI = 3.14159265359 (rkdg_swe_bc_tide.hpp:73-100, rkdg_swe_bc_flow.hpp:72-102), in FP64
// in both precisions. Out of line: only the extra CTAs of a step's last stage come here.
static __device__ __noinline__ void form_step_time(const TimeArgs* Tp, int block) {
    const TimeArgs& T = *Tp;
    const double t = T.cur ? T.cur->t + T.dt : T.t0;  // ESSPRKStepper::operator++ (:55-58)
    if (block == 0) {
        const int s = threadIdx.x;
        if (s < T.nstages) {
            T.next->at[s].ft = dgsw_fn_prepare(T.fn_set, T.fn_params, t + T.off[s]);
            if (T.fn_set == DGSW_FN_MANUFACTURED_SINE) sine_constants(T.fn_params, T.next->at[s]);
        }
        if (s == 0) {
            T.next->t = t;
            T.next->step = T.cur ? T.cur->step + 1 : T.step0;
        }
        return;
    }
    const int per_set = T.n_forced * T.ng;
    const int i = (block - 1) * (int)blockDim.x + (int)threadIdx.x;
    if (i >= T.nsets * per_set) return;
    constexpr double REF_PI = 3.14159265359;
    const int set = i / per_set, gp = i % T.ng;
    const double ts = t + T.off[T.set_stage[set]];
    const double ramp = forcing_ramp(T, ts);
    const int2 fc = T.fface[(i % per_set) / T.ng];
    double acc = 0.0;
    for (int c = 0; c < fc.y; ++c) {
        const double* r = T.fcon + (size_t)(fc.x + c) * FORCE_STRIDE_DEV;
        acc += ramp * r[1] * r[3 + gp] * cos(r[0] * ts + (r[2] - r[6 + gp]) * REF_PI / 180.0);
    }
    T.fval[i] = acc;
}
// CTAs of `threads` threads that form_step_time takes
inline int step_time_blocks(const TimeArgs& T, int threads) {
    return 1 + (T.nsets * T.n_forced * T.ng + threads - 1) / threads;
}

// Real is the arithmetic type of the stage (FP32 bulk or FP64); the stage states and stored stage
// solutions are FP64 in both, so that the RK update does not accumulate FP32 rounding from stage to stage
template <typename Real>
struct StageArgs {
    const double* qk[DGSW_RK_MAX_STAGES];  // stage states used by this stage's combination, q_s last
    const double* solk[DGSW_RK_MAX_STAGES];
    double a[DGSW_RK_MAX_STAGES];
    double bdt[DGSW_RK_MAX_STAGES];
    int nterms;
    int store_sol;  // write sol_s (needed when a later stage uses it)
    double* q_out;
    double* sol_out;
    const Real* bath;           // [3][ne_pad] bathymetry modes of the linear part
    const Real* geo;            // [4][ne_pad] J^-1(0,0), J^-1(0,1), J^-1(1,0), J^-1(1,1)
    const int* enodes;          // [3][ne_pad]
    // per face: kind (bits 0-2, EdgeKind) | the element is the interface's in side (bit 3) | payload << 4: the trace
    // slot across the face (a neighbour's, or the boundary face's ghost slot), or the levee interface's index
    const int* fmeta;           // [3][ne_pad]
    const Real* fw;             // [3][ne_pad] half the face's length over the element's |J|
    const int2* tiles;          // per tile: offset into halo, halo faces
    const int2* halo;           // tile lists: (element, face) per halo face, then (forcing record, 0) per boundary face
    const double2* xy;          // node coordinates
    const double* nz;           // node bathymetry depth (wet/dry vertex depths)
    const unsigned char* wet_in;
    unsigned char* wet_out;
    const int* ref_of_dev;
    double* baryctr;  // [3][ne_pad] barycentre values of the new state for the slope limiter, or null
    DevStatus* status;
    const DevClock* clock;  // this step's copy
    TimeArgs time;          // the next step's copy, formed by `n_time` extra CTAs of the last stage's launch
    int n_time;
    int ntiles;
    int stage_index, nstages;  // this stage and the stages per step (the NaN report's stage counter)
    int ne;
    int ne_pad;
    double g;
    double h_o, h_o_thr;
    int fn_set;
    double fn_params[16];
    int spherical;
    const Real* sph;  // [spherical_rows][ne_pad] spherical correction factors (null without)
    // bottom friction (swe_source.hpp:29-51): DGSW_FRICTION_NONE / CHEZY / MANNING
    int friction;
    double friction_cf;
    const Real* manning;  // [ne_pad] g n^2 per element (Manning)
    const double* fval;   // [n_forced][NG] this stage's tide / flow values at the forced faces' Gauss points
    // levee interface fluxes of this stage, [n_levee][2][3][NG] (levee.cu): in side, then ex side; zero where both
    // sides are dry
    const double* levF;
    unsigned char* went_dry;  // [ne] wet_dry_state.went_completely_dry of the last wet/dry pass, or null
    int reverse;              // visit the tiles in reverse order (grid = one CTA per tile)
    // Stage increments (the SPLIT kernels, FP32 arithmetic without wetting/drying, limiter or levees): the
    // carried state q_0 is kept compensated, as the unevaluated sum q0f + q0lo of two Real values (q0f the
    // rounding of q_0, q0lo the rounding of the remainder: a 48-bit significand), and each intermediate
    // stage state as its increment d_s = q_s - q_0 in Real. With sum_k a_sk = 1 the combination
    // q_{s+1} = sum_k a_sk q_k + dt b_sk L(q_k) becomes d_{s+1} = sum_k a_sk d_k + dt b_sk L(q_k) (d_0 = 0):
    // q_0 leaves it, so the increments round relative to their own small size. The last stage forms
    // q0f + q0lo + d_ns in FP64 and splits it again.
    const Real* dk[DGSW_RK_MAX_STAGES];     // increments of the combination's terms (null for q_0), d_s last
    const Real* dsolk[DGSW_RK_MAX_STAGES];  // stored stage solutions of the earlier terms, in Real
    const Real* q0f;                        // carried state, leading part: stage input q_s = q0f + d_s
    const Real* q0lo;                       // carried state, trailing part (read by the last stage)
    Real* d_out;                            // d_{s+1} (intermediate stages)
    Real* dsol_out;                         // this stage's solution, when a later stage reads it
    Real* q0f_out;                          // new carried state, leading part (last stage)
    Real* q0lo_out;                         // new carried state, trailing part (last stage)
    int last;                               // this is the step's last stage
};

// ------------------------------------------------------------------------------------------------
// LLF flux, rkdg_swe_LLF_flux.hpp:7-60 (sp applied to the in-side normal flux only, as there)
// ------------------------------------------------------------------------------------------------
template <typename Real>
__device__ __forceinline__ void llf_flux(Real gravity, const Real qin[3], const Real qex[3], Real bath, Real sp,
                                         Real nx, Real ny, Real F[3]) {
    const Real h_in = qin[0] + bath;
    const Real ih_in = Real(1) / h_in;
    const Real u_in = qin[1] * ih_in;
    const Real v_in = qin[2] * ih_in;
    const Real h_ex = qex[0] + bath;
    const Real ih_ex = Real(1) / h_ex;
    const Real u_ex = qex[1] * ih_ex;
    const Real v_ex = qex[2] * ih_ex;
    const Real un_in = u_in * nx + v_in * ny;
    const Real un_ex = u_ex * nx + v_ex * ny;
    const Real spc = (nx * sp) * (nx * sp) + ny * ny;
    const Real lam = fmax(fabs(un_in) + sqrt(gravity * h_in * spc), fabs(un_ex) + sqrt(gravity * h_ex * spc));
    const Real pe_in = gravity * (qin[0] * qin[0] * Real(0.5) + qin[0] * bath);
    const Real pe_ex = gravity * (qex[0] * qex[0] * Real(0.5) + qex[0] * bath);
    const Real uuh_in = u_in * qin[1], vvh_in = v_in * qin[2], uvh_in = u_in * qin[2];
    const Real uuh_ex = u_ex * qex[1], vvh_ex = v_ex * qex[2], uvh_ex = u_ex * qex[2];
    const Real f0 = sp * qin[1] * nx + qin[2] * ny;
    const Real f1 = sp * (uuh_in + pe_in) * nx + uvh_in * ny;
    const Real f2 = sp * uvh_in * nx + (vvh_in + pe_in) * ny;
    const Real e0 = qex[1] * nx + qex[2] * ny;
    const Real e1 = (uuh_ex + pe_ex) * nx + uvh_ex * ny;
    const Real e2 = uvh_ex * nx + (vvh_ex + pe_ex) * ny;
    F[0] = Real(0.5) * (f0 + e0 + lam * (qin[0] - qex[0]));
    F[1] = Real(0.5) * (f1 + e1 + lam * (qin[1] - qex[1]));
    F[2] = Real(0.5) * (f2 + e2 + lam * (qin[2] - qex[2]));
}

// One side of a face at a Gauss point: the trace, 1 / h and the wave speed sqrt(g h)
template <typename Real>
struct Side {
    Two<Real> q;  // qx, qy
    Real ze, b, ih, c;
};
template <typename Real>
__device__ __forceinline__ void complete(Side<Real>& s, Real g) {
    const Real h = s.ze + s.b;
    s.ih = Real(1) / h;
    s.c = sqrt(g * h);
}

// The LLF flux above (sp = 1) of the own side towards the neighbour n, doubled and times w, along the own
// outward normal times w, N = w nrm: with qn = q . N and un = qn / h the normal flux of a side is
// (qn, q un + pe N), the same terms as above with the products regrouped (a few ulps). Every term changes sign
// exactly when the sides trade places and the same N turns round.
template <bool PK, typename Real>
__device__ __forceinline__ void llf_sides(Real g, const Side<Real>& o, const Side<Real>& n, Two<Real> N, Real w, Real& F0,
                                          Two<Real>& F12) {
    const Real fo = fma_rn(o.q.x, N.x, mul_rn(o.q.y, N.y)), fn = fma_rn(n.q.x, N.x, mul_rn(n.q.y, N.y));
    const Real uo = mul_rn(fo, o.ih), un = mul_rn(fn, n.ih);
    const Real po = mul_rn(mul_rn(g, o.ze), fma_rn(Real(0.5), o.ze, o.b));
    const Real pn = mul_rn(mul_rn(g, n.ze), fma_rn(Real(0.5), n.ze, n.b));
    const Two<Real> go = fma2<PK, Real>(o.q, uo, mul2<PK, Real>(N, po));
    const Two<Real> gn = fma2<PK, Real>(n.q, un, mul2<PK, Real>(N, pn));
    const Real lam = fmax(fma_rn(o.c, w, fabs(uo)), fma_rn(n.c, w, fabs(un)));
    F0 = fma_rn(lam, add_rn(o.ze, -n.ze), add_rn(fo, fn));
    F12 = fma2<PK, Real>(add2<PK, Real>(o.q, Two<Real>{-n.q.x, -n.q.y}), lam, add2<PK, Real>(go, gn));
}

// Outward normal of face f times w = (half its length) / |J|: a face's normal is along the gradient of the
// opposite vertex' barycentric coordinate, and with that length the rows of J^-1 are the vectors themselves
template <typename Real>
__device__ __forceinline__ Two<Real> scaled_normal(int f, Real Ji00, Real Ji01, Real Ji10, Real Ji11) {
    if (f == 0) return {Ji00 + Ji10, Ji01 + Ji11};
    if (f == 1) return {-Ji00, -Ji01};
    return {-Ji10, -Ji11};
}

// Wet/dry fix-ups of ISP::Internal (rkdg_swe_is_internal.hpp:47-90) for an interface with one dry side whose LLF
// ze-flux exceeds 1e-12 in magnitude, as the own side sees them: F0, F12 is its flux towards n (llf_sides: doubled,
// times w) before and after. The reference's two branches by the flux's sign are one here, since a side's flux is
// negative where the other's is positive: water leaves a dry element (none does), or comes from a dry neighbour (none
// does, a reflective wall), or flows into a dry element (without gravity).
template <bool PK, typename Real>
__device__ __forceinline__ void wd_fixup(Real g, Side<Real> o, Side<Real> n, Two<Real> N, Real w, bool wet, bool wn, Real& F0,
                                         Two<Real>& F12) {
    const Real iw = Real(1) / w, thr = Real(2e-12) * w;
    if (F0 > thr) {
        if (!wet) F0 = Real(0), F12 = {Real(0), Real(0)};
    } else if (F0 < -thr) {
        if (!wn) {
            // the mirrored state's flux (rkdg_swe_bc_land.hpp:68-86) in closed form: no mass through the wall, and twice
            // the pressure and the normal momentum's upwinding on it
            const Real fo = fma_rn(o.q.x, N.x, mul_rn(o.q.y, N.y)), uo = fo * o.ih;
            const Real a = (uo + fabs(uo) + o.c * w) * (2 * fo * iw * iw) + 2 * (g * o.ze * (Real(0.5) * o.ze + o.b));
            F0 = Real(0), F12 = {a * N.x, a * N.y};
        } else {
            o.c = n.c = Real(0);
            Real F0g;
            llf_sides<PK, Real>(Real(0), o, n, N, w, F0g, F12);
        }
    }
}

// three values returned by value from the out-of-line helpers below: an output array passed by
// address would live in local memory at every call site
template <typename Real>
struct Val3 {
    Real v0, v1, v2;
};

// analytic function sets evaluated out of line (one copy per kernel); T: the stage's time factors
template <typename Real>
__device__ __noinline__ Val3<Real> fn_eval_dev(int id, const double* P, const dgsw_fn_time* T, int source, Real x,
                                               Real y) {
    Real out[3];
    dgsw_fn_eval<Real>(id, P, *T, source, x, y, out);
    return Val3<Real>{out[0], out[1], out[2]};
}

// the Manning friction factor g n^2 / h^(1/3), bounded below by the Chezy coefficient (swe_source.hpp:37-42);
// h^(-1/3) through the reciprocal cube root (the reference's pow(h, 1/3) differs from cbrt by the
// rounding of 1/3, a few ulps)
template <typename Real>
__device__ __forceinline__ Real manning_cf(Real gn2, Real h, Real cf0) {
    Real cf = gn2 * rcbrt(h);
    if (cf < cf0) cf = cf0;
    return cf;
}

// The manufactured sine set's source terms inline, with its constants of the stage (sine_constants); every
// other set goes through fn_eval_dev.
template <typename Real>
struct SineSrc {
    Real k, c1, c2, c3, c5, c6, c0, g, H, kpi;
};

template <typename Real>
__device__ __forceinline__ SineSrc<Real> sine_src_load(const StageTime& T) {
    const Real* c;
    if constexpr (sizeof(Real) == 8)
        c = T.sine;
    else
        c = T.sine_f;
    return SineSrc<Real>{c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9]};
}

// sin and cos of k x: FP64 through sincospi(2 x / L), whose argument reduction is an exact rounding to an
// integer (sincos reduces by pi in several parts; the two differ by the rounding of 2 pi / L, a few 1e-16
// relative); FP32 through the range-reduced hardware sine/cosine
template <typename Real>
__device__ __forceinline__ void sine_src_sincos(const SineSrc<Real>& S, Real x, Real& s, Real& c) {
    if constexpr (sizeof(Real) == 8)
        sincospi(S.kpi * x, &s, &c);
    else
        dgsw_sincos(S.k * x, &s, &c);
}

// sin and cos of an angle a0 + e from s0 = sin a0, c0 = cos a0 and a small increment e (|e| <= 0.05), by the
// angle-addition identities with the Taylor series of sin e and cos e through e^9 / e^8 (remainder below
// 1e-19). FP64 elements evaluate sin and cos at their centroid and turn them to the quadrature points
// this way.
__device__ __forceinline__ void rotate_small(double s0, double c0, double e, double& s, double& c) {
    const double z = e * e;
    const double ce = 1.0 + z * (-1.0 / 2 + z * (1.0 / 24 + z * (-1.0 / 720 + z * (1.0 / 40320))));
    const double se = e * (1.0 + z * (-1.0 / 6 + z * (1.0 / 120 + z * (-1.0 / 5040 + z * (1.0 / 362880)))));
    s = s0 * ce + c0 * se;
    c = c0 * ce - s0 * se;
}

// the set's source at a point from sin / cos of k x and k y: the terms of fn_sine_source regrouped,
// S_x = qx_t + (3 qx qxx + qxy qy) / h - qx (qx zex + qy zey) / h^2 + g h zex (qyy = qxx), S_y likewise
template <bool PK, typename Real>
__device__ __forceinline__ void sine_src_terms(const SineSrc<Real>& S, Real sx, Real cx, Real sy, Real cy, Real& s0,
                                               Two<Real>& s12) {
    const Real Pp = sx * cy, Sq = cx * sy;
    const Two<Real> QR = {cx * cy, sx * sy};
    const Two<Real> q = mul2<PK, Real>(QR, Two<Real>{-S.c2, S.c2});    // qx, qy
    const Two<Real> zd = mul2<PK, Real>(QR, Two<Real>{S.c3, -S.c3});   // zex, zey
    const Real qxx3 = (Real(3) * S.c5) * Pp, qxy = S.c5 * Sq;
    const Real h = S.c1 * Pp + S.H;
    const Real ih = Real(1) / h;
    const Real D = (q.x * zd.x + q.y * zd.y) * ih;
    const Two<Real> t = fma2<PK, Real>(q, qxx3, mul2<PK, Real>(Two<Real>{q.y, q.x}, qxy));
    const Two<Real> a = fma2<PK, Real>(zd, S.g * h, mul2<PK, Real>(QR, Two<Real>{-S.c6, S.c6}));
    s0 = S.c0 * Pp;
    s12 = fma2<PK, Real>(fma2<PK, Real>(q, -D, t), ih, a);
}

template <bool PK, typename Real>
__device__ __forceinline__ void sine_src_eval(const SineSrc<Real>& S, Real x, Real y, Real& s0, Two<Real>& s12) {
    Real sx, cx, sy, cy;
    sine_src_sincos<Real>(S, x, sx, cx);
    sine_src_sincos<Real>(S, y, sy, cy);
    sine_src_terms<PK, Real>(S, sx, cx, sy, cy, s0, s12);
}

// the sine set's source at one point, out of line
template <typename Real>
__device__ __noinline__ Val3<Real> sine_src_far(const StageTime* T, Real x, Real y) {
    const SineSrc<Real> S = sine_src_load<Real>(*T);
    Real s0;
    Two<Real> s12;
    sine_src_eval<false, Real>(S, x, y, s0, s12);
    return Val3<Real>{s0, s12.x, s12.y};
}

// ------------------------------------------------------------------------------------------------
// wetting/drying of one p>=1 element on its vertex values, swe_post_wet_dry.hpp:6-145, in FP64.
// qv: modal state (first three modes carry the linear part); returns the new wet flag and writes
// the new modes back (higher modes are zeroed whenever the vertex values are re-projected, like
// ProjectLinearToBasis).
// ------------------------------------------------------------------------------------------------
template <int ND, typename Real>
__device__ __forceinline__ bool wetting_drying(Real (&qv)[3][ND], const double bv[3], double bath_min, double h_o,
                                               double thr, bool wet, bool& went_dry) {
    double z[3], qx[3], qy[3], h[3];
    // ProjectBasisToLinear through T_basis_linear (basis_dubiner_2D.cpp:213-234)
    {
        const double a = qv[0][0], b = qv[0][1], c = qv[0][2];
        z[0] = a - b - c;
        z[1] = a - b + c;
        z[2] = a + 2.0 * b;
        const double ax = qv[1][0], bx = qv[1][1], cx = qv[1][2];
        qx[0] = ax - bx - cx;
        qx[1] = ax - bx + cx;
        qx[2] = ax + 2.0 * bx;
        const double ay = qv[2][0], by = qv[2][1], cy = qv[2][2];
        qy[0] = ay - by - cy;
        qy[1] = ay - by + cy;
        qy[2] = ay + 2.0 * by;
    }
    int ndry = 0;
    for (int v = 0; v < 3; ++v) {
        h[v] = z[v] + bv[v];
        if (h[v] <= h_o + thr) ++ndry;
    }
    double h_avg = (0.0 + h[0] + h[1] + h[2]) / 3;
    went_dry = h_avg <= thr;  // wet_dry_state.went_completely_dry
    if (h_avg <= thr) h_avg = thr;
    bool reproject = false, check = false;
    if (ndry == 0) {
        if (wet) return true;
        check = true;
    } else if (ndry == 3) {
        for (int v = 0; v < 3; ++v) {
            z[v] = h_avg - bv[v];
            qx[v] = 0.0;
            qy[v] = 0.0;
        }
        wet = false;
        reproject = true;
    } else {
        if (h_avg <= h_o + thr) {
            for (int v = 0; v < 3; ++v) {
                z[v] = h_avg - bv[v];
                qx[v] = 0.0;
                qy[v] = 0.0;
            }
        } else {
            // first minimum / first maximum, like std::min_element / std::max_element (the values
            // are tracked beside the indices: an array indexed at run time would live in local memory;
            // here some vertices are dry and some are not, so hmin != hmax)
            int hmin = 0, hmax = 0;
            double hminv = h[0], hmaxv = h[0];
#pragma unroll
            for (int v = 1; v < 3; ++v) {
                if (h[v] < hminv) hmin = v, hminv = h[v];
                if (h[v] > hmaxv) hmax = v, hmaxv = h[v];
            }
            const int hmid = 3 - hmax - hmin;
            const double hmidv = hmid == 0 ? h[0] : (hmid == 1 ? h[1] : h[2]);
            const double tmin = h_o;
            const double tmid = fmax(h_o, hmidv - (tmin - hminv) / 2);
            const double tmax = hmaxv - (tmin - hminv) - (tmid - hmidv);
#pragma unroll
            for (int v = 0; v < 3; ++v) h[v] = v == hmin ? tmin : (v == hmax ? tmax : tmid);
            double dqx = 0, dqy = 0;
            int ndv = 0;
            for (int v = 0; v < 3; ++v)
                if (h[v] <= h_o + thr) {
                    ndv++;
                    dqx += qx[v];
                    dqy += qy[v];
                    qx[v] = 0.0;
                    qy[v] = 0.0;
                }
            for (int v = 0; v < 3; ++v) {
                z[v] = h[v] - bv[v];
                if (h[v] > h_o + thr) {
                    qx[v] += dqx / (3 - ndv);
                    qy[v] += dqy / (3 - ndv);
                }
            }
        }
        reproject = true;
        check = true;
    }
    if (check) {
        // z at the first maximum of h
        double hmaxv = h[0], zmax = z[0];
#pragma unroll
        for (int v = 1; v < 3; ++v)
            if (h[v] > hmaxv) hmaxv = h[v], zmax = z[v];
        if (zmax > h_o - bath_min) {
            wet = true;
        } else {
            wet = false;
            for (int v = 0; v < 3; ++v) {
                qx[v] = 0.0;
                qy[v] = 0.0;
            }
            reproject = true;
        }
    }
    if (reproject) {
        // ProjectLinearToBasis through T_linear_basis (:236-257)
        auto project = [&](const double (&s)[3], int var) {
            qv[var][0] = (Real)(s[0] * (1.0 / 3.0) + s[1] * (1.0 / 3.0) + s[2] * (1.0 / 3.0));
            qv[var][1] = (Real)(s[0] * (-1.0 / 6.0) + s[1] * (-1.0 / 6.0) + s[2] * (1.0 / 3.0));
            qv[var][2] = (Real)(s[0] * (-1.0 / 2.0) + s[1] * (1.0 / 2.0));
#pragma unroll
            for (int k = 3; k < ND; ++k) qv[var][k] = Real(0);
        };
        project(z, 0);
        project(qx, 1);
        project(qy, 2);
    }
    return wet;
}

// ------------------------------------------------------------------------------------------------
// compile-time table access
// ------------------------------------------------------------------------------------------------
template <int P>
using MT = ct::Master<P>;

// trace of an element's face F at the edge Gauss points: ze, qx, qy and bathymetry (the levee and trouble passes)
template <int P, int F, typename Real>
__device__ __forceinline__ void face_trace(const Real (&q)[3][MT<P>::ND], const Real (&b)[3],
                                           Real (&t)[4][MT<P>::NG]) {
    constexpr int ND = MT<P>::ND, NG = MT<P>::NG;
    sfor<0, NG>([&](auto G) {
        constexpr int g = decltype(G)::value;
        sfor<0, 3>([&](auto V) {
            constexpr int v = decltype(V)::value;
            Real s = Real(0);
            sfor<0, ND>([&](auto K) {
                constexpr int k = decltype(K)::value;
                constexpr double c = MT<P>::fphi((F * ND + k) * NG + g);
                if constexpr (c != 0.0) s += q[v][k] * (Real)c;
            });
            t[v][g] = s;
        });
        Real sb = Real(0);
        sfor<0, 3>([&](auto K) {
            constexpr int k = decltype(K)::value;
            constexpr double c = MT<P>::fphi((F * ND + k) * NG + g);
            if constexpr (c != 0.0) sb += b[k] * (Real)c;
        });
        t[3][g] = sb;
    });
}

// Trace slots in shared memory, 16-byte vectors [vector][NS slots]: FP32 one vector (qx, qy, ze, b) per Gauss
// point; FP64 three, (qx, qy), (ze, b) and (1 / h, sqrt(g h)), so that the divisions and square roots are
// taken once per trace and not by both sides. A thread's slots are three apart: its 16-byte accesses meet
// the banks without conflicts.
template <int P, typename Real>
struct Trace {
    static constexpr int NG = MT<P>::NG;
    static constexpr int NV = sizeof(Real) == 8 ? 3 : 1;  // vectors per Gauss point
    static __device__ __forceinline__ void put(unsigned char* tr, int NS, int slot, int gp, const Side<Real>& s) {
        if constexpr (sizeof(Real) == 4) {
            reinterpret_cast<float4*>(tr)[gp * NS + slot] = make_float4(s.q.x, s.q.y, s.ze, s.b);
        } else {
            double2* v = reinterpret_cast<double2*>(tr) + gp * NV * NS + slot;
            v[0] = make_double2(s.q.x, s.q.y);
            v[NS] = make_double2(s.ze, s.b);
            v[2 * NS] = make_double2(s.ih, s.c);
        }
    }
    static __device__ __forceinline__ Side<Real> get(const unsigned char* tr, int NS, int slot, int gp, Real g) {
        Side<Real> s;
        if constexpr (sizeof(Real) == 4) {
            const float4 v = reinterpret_cast<const float4*>(tr)[gp * NS + slot];
            s.q = {v.x, v.y}, s.ze = v.z, s.b = v.w;
            complete<Real>(s, g);
        } else {
            const double2* v = reinterpret_cast<const double2*>(tr) + gp * NV * NS + slot;
            const double2 a = v[0], b = v[NS], c = v[2 * NS];
            s.q = {a.x, a.y}, s.ze = b.x, s.b = b.y, s.ih = c.x, s.c = c.y;
        }
        return s;
    }
};

// the trace of an element's face F at Gauss point G: sums over the modes in ascending order (the same
// arithmetic for tile and halo elements)
template <int P, int F, int G, bool PK, typename Real>
__device__ __forceinline__ Side<Real> face_point(const Real (&q)[3][MT<P>::ND], const Real (&b)[3]) {
    constexpr int ND = MT<P>::ND, NG = MT<P>::NG;
    Two<Real> s12 = {Real(0), Real(0)}, s0b = {Real(0), Real(0)};
    sfor<0, ND>([&](auto K) {
        constexpr int k = decltype(K)::value;
        constexpr double c = MT<P>::fphi((F * ND + k) * NG + G);
        if constexpr (counts(c)) {
            s12 = fma2<PK, Real>(Two<Real>{q[1][k], q[2][k]}, (Real)c, s12);
            if constexpr (k < 3)
                s0b = fma2<PK, Real>(Two<Real>{q[0][k], b[k]}, (Real)c, s0b);
            else
                s0b.x = fma_rn(q[0][k], (Real)c, s0b.x);
        }
    });
    Side<Real> s;
    s.q = s12, s.ze = s0b.x, s.b = s0b.y, s.ih = s.c = Real(0);
    return s;
}
// `whole` false: a dry element's face in a wet/dry kernel, whose 1 / h and sqrt(g h) only the interfaces with one
// dry side would read; they form it themselves
template <int P, int F, bool PK, typename Real>
__device__ __forceinline__ void put_face(unsigned char* tr, int NS, int slot, const Real (&q)[3][MT<P>::ND],
                                         const Real (&b)[3], Real g, bool whole) {
    sfor<0, MT<P>::NG>([&](auto G) {
        constexpr int gp = decltype(G)::value;
        Side<Real> s = face_point<P, F, gp, PK, Real>(q, b);
        if (sizeof(Real) == 8 && whole) complete<Real>(s, g);
        Trace<P, Real>::put(tr, NS, slot, gp, s);
    });
}

// the same for a face known only at run time, with the face's basis values from a [mode][gp] table: the halo
// faces of a warp belong to different faces, and one compile-time copy per face would split the warp.
// Entries that are zero on this face but not on another add a zero product (the sum is unchanged), so the
// values equal put_face's bit for bit.
template <int P, bool PK, typename Real>
__device__ __forceinline__ void put_face_rt(unsigned char* tr, int NS, int slot, const Real (&q)[3][MT<P>::ND],
                                            const Real (&b)[3], const Real* cf, Real g) {
    constexpr int ND = MT<P>::ND, NG = MT<P>::NG;
    sfor<0, NG>([&](auto G) {
        constexpr int gp = decltype(G)::value;
        Two<Real> s12 = {Real(0), Real(0)}, s0b = {Real(0), Real(0)};
        sfor<0, ND>([&](auto K) {
            constexpr int k = decltype(K)::value;
            constexpr bool used = counts(MT<P>::fphi((0 * ND + k) * NG + gp)) ||
                                  counts(MT<P>::fphi((1 * ND + k) * NG + gp)) ||
                                  counts(MT<P>::fphi((2 * ND + k) * NG + gp));
            if constexpr (used) {
                const Real c = cf[k * NG + gp];
                s12 = fma2<PK, Real>(Two<Real>{q[1][k], q[2][k]}, c, s12);
                if constexpr (k < 3)
                    s0b = fma2<PK, Real>(Two<Real>{q[0][k], b[k]}, c, s0b);
                else
                    s0b.x = fma_rn(q[0][k], c, s0b.x);
            }
        });
        Side<Real> s;
        s.q = s12, s.ze = s0b.x, s.b = s0b.y;
        if constexpr (sizeof(Real) == 8) complete<Real>(s, g);
        Trace<P, Real>::put(tr, NS, slot, gp, s);
    });
}

// A boundary face's ghost states into its trace slot, at the Gauss points as a neighbour across the face
// would number them; out of line (boundary elements only). own: the face's own trace slot.
// BC::Land: normal momentum mirrored (rkdg_swe_bc_land.hpp:44-56); BC::Function: ic_q(t, x_gp)
// (rkdg_swe_bc_function.hpp:33-50); BC::Tide and BC::Flow (rkdg_swe_bc_tide.hpp:73-100,
// rkdg_swe_bc_flow.hpp:72-102) from the stage's forcing values (form_step_time): a tide sets the ghost
// surface elevation and keeps the interior momentum; a flow keeps the interior elevation and sets the ghost
// momentum to the value times the outward normal. All of them keep the interior bathymetry.
template <int P, typename Real>
__device__ __noinline__ void ghost_face(const StageArgs<Real>* Ap, unsigned char* tr, int NS, int own, int slot, int d,
                                        int f, int kind, int forcing, Real Nx, Real Ny,
                                        Real w) {
    const Real iw = Real(1) / w, nx = Nx * iw, ny = Ny * iw;
    const StageArgs<Real>& A = *Ap;
    constexpr int NG = MT<P>::NG;
    const Real g = (Real)A.g;
    double xa = 0, ya = 0, xb = 0, yb = 0;
    if (kind == 2) {
        // the Gauss points lie on the segment from node (f+1)%3 to node (f+2)%3
        const double2 pa = A.xy[A.enodes[((f + 1) % 3) * A.ne_pad + d]];
        const double2 pb = A.xy[A.enodes[((f + 2) % 3) * A.ne_pad + d]];
        xa = pa.x, ya = pa.y, xb = pb.x, yb = pb.y;
    }
    sfor<0, NG>([&](auto GP) {
        constexpr int gp = decltype(GP)::value;
        constexpr double wa = MT<P>::fpsi((0 * 3 + 1) * NG + gp), wb = MT<P>::fpsi((0 * 3 + 2) * NG + gp);
        Side<Real> s = Trace<P, Real>::get(tr, NS, own, gp, g);
        if (kind == 1) {
            const Real tx = -ny, ty = nx;
            const Real qn = -(s.q.x * nx + s.q.y * ny);
            const Real qt = s.q.x * tx + s.q.y * ty;
            s.q = {qn * nx + qt * tx, qn * ny + qt * ty};
        } else if (kind == 2) {
            Real qe[3];
            dgsw_fn_eval<Real>(A.fn_set, A.fn_params, A.clock->at[A.stage_index].ft, 0, (Real)(xa * wa + xb * wb),
                               (Real)(ya * wa + yb * wb), qe);
            s.ze = qe[0], s.q = {qe[1], qe[2]};
        } else {
            const Real v = (Real)A.fval[forcing * NG + gp];
            if (kind == 4)
                s.q = {v * nx, v * ny};
            else
                s.ze = v;
        }
        // FP64: the other kinds keep the interior depth, whose 1 / h and sqrt(g h) came with the own trace
        if (sizeof(Real) == 8 && (kind == 2 || kind == 3)) complete<Real>(s, g);
        Trace<P, Real>::put(tr, NS, slot, NG - 1 - gp, s);
    });
}

// The spherical correction cos(phi_0) / cos(y / R) at an element's face and volume Gauss points (geometry alone):
// rows face * NG + gp, then 3 NG + gp, of [ne_pad] values, formed once per handle. In the stage kernel it was a cosine in
// FP64 per point, and two per face point as both elements of a face evaluate its flux. 8 steps of 131,072 triangles:
// tidal channel p = 1 FP64 0.71 -> 0.38 ms, FP32 0.43 -> 0.28, p = 2 FP64 2.09 -> 1.29, FP32 0.99 -> 0.64; wet/dry bowl
// p = 1 FP64 0.76 -> 0.38, FP32 0.39 -> 0.24.
template <int P>
constexpr int spherical_rows() {
    return 3 * MT<P>::NG + MT<P>::NQ;
}
template <int P, typename Real>
__global__ void __launch_bounds__(128) spherical_kernel(const int* __restrict__ enodes, const double2* __restrict__ xy,
                                                        double cos_lat0, double R, int ne, int ne_pad,
                                                        Real* __restrict__ sph) {
    constexpr int NG = MT<P>::NG, NQ = MT<P>::NQ;
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= ne) return;
    double y[3];
    sfor<0, 3>([&](auto V) { y[decltype(V)::value] = xy[enodes[decltype(V)::value * ne_pad + d]].y; });
    sfor<0, 3>([&](auto F) {
        constexpr int f = decltype(F)::value;
        sfor<0, NG>([&](auto G) {
            constexpr int g = decltype(G)::value;
            constexpr double wa = MT<P>::fpsi((0 * 3 + 1) * NG + g), wb = MT<P>::fpsi((0 * 3 + 2) * NG + g);
            sph[(size_t)(f * NG + g) * ne_pad + d] = (Real)(cos_lat0 / cos((y[(f + 1) % 3] * wa + y[(f + 2) % 3] * wb) / R));
        });
    });
    sfor<0, NQ>([&](auto Q) {
        constexpr int q = decltype(Q)::value;
        constexpr Real p0 = (Real)MT<P>::psi(0 * NQ + q), p1 = (Real)MT<P>::psi(1 * NQ + q), p2 = (Real)MT<P>::psi(2 * NQ + q);
        sph[(size_t)(3 * NG + q) * ne_pad + d] = (Real)(cos_lat0 / cos((y[0] * p0 + y[1] * p1 + y[2] * p2) / R));
    });
}

// llf_sides with the spherical correction: sp multiplies the x component of the in side's normal flux and of the normal in
// both sides' wave speeds (llf_flux, the products regrouped as in llf_sides)
template <bool PK, typename Real>
__device__ __forceinline__ void llf_sides_spherical(Real g, const Side<Real>& o, const Side<Real>& n, Two<Real> N, Real sp,
                                                    bool is_in, Real& F0, Two<Real>& F12) {
    const Real nxs = sp * N.x;
    const Real W = sqrt(fma_rn(nxs, nxs, mul_rn(N.y, N.y)));
    const Two<Real> No = {is_in ? nxs : N.x, N.y}, Nn = {is_in ? N.x : nxs, N.y};
    const Real fo = fma_rn(o.q.x, No.x, mul_rn(o.q.y, No.y)), fn = fma_rn(n.q.x, Nn.x, mul_rn(n.q.y, Nn.y));
    const Real po = mul_rn(mul_rn(g, o.ze), fma_rn(Real(0.5), o.ze, o.b));
    const Real pn = mul_rn(mul_rn(g, n.ze), fma_rn(Real(0.5), n.ze, n.b));
    const Two<Real> go = fma2<PK, Real>(o.q, mul_rn(fo, o.ih), mul2<PK, Real>(No, po));
    const Two<Real> gn = fma2<PK, Real>(n.q, mul_rn(fn, n.ih), mul2<PK, Real>(Nn, pn));
    const Real uo = mul_rn(fma_rn(o.q.x, N.x, mul_rn(o.q.y, N.y)), o.ih), un = mul_rn(fma_rn(n.q.x, N.x, mul_rn(n.q.y, N.y)), n.ih);
    const Real lam = fmax(fma_rn(o.c, W, fabs(uo)), fma_rn(n.c, W, fabs(un)));
    F0 = fma_rn(lam, add_rn(o.ze, -n.ze), add_rn(fo, fn));
    F12 = fma2<PK, Real>(add2<PK, Real>(o.q, Two<Real>{-n.q.x, -n.q.y}), lam, add2<PK, Real>(go, gn));
}

// wd_fixup with the spherical correction: the own side is the in side of the wall's and of the gravity-free flux, and the
// wall's mass flux, whose two halves no longer cancel, stays (as in the reference)
template <bool PK, typename Real>
__device__ __forceinline__ void wd_fixup_spherical(Real g, Side<Real> o, Side<Real> n, Two<Real> N, Real w, Real sp, bool wet,
                                                   bool wn, Real& F0, Two<Real>& F12) {
    const Real thr = Real(2e-12) * w;
    if (F0 > thr) {
        if (!wet) F0 = Real(0), F12 = {Real(0), Real(0)};
    } else if (F0 < -thr) {
        Real Fw;
        if (!wn) {  // the neighbour is the own state mirrored
            const Real a = Real(-2) * fma_rn(o.q.x, N.x, mul_rn(o.q.y, N.y)) / (w * w);
            n = o;
            n.q = fma2<PK, Real>(N, a, o.q);
        } else {
            g = o.c = n.c = Real(0);
        }
        llf_sides_spherical<PK, Real>(g, o, n, N, sp, true, Fw, F12);
        if (!wn) F0 = Fw;
    }
}

// A face Gauss point where the spherical correction applies: the doubled flux times w of the own side, wet/dry fix-ups
// included. Out of line and without calls of its own, so that the kernel's registers are those of a run without the
// correction and none are saved here (with a call inside, 20 % of an FP64 stage of 8,192 triangles went into saving them).
template <int P, bool WD, typename Real>
__device__ __noinline__ Val3<Real> spherical_point(const StageArgs<Real>* Ap, const unsigned char* tr, int NS, int own,
                                                   int slot, int gp, Real sp, bool is_in, bool wet, bool wn, Real Nx,
                                                   Real Ny, Real w) {
    constexpr bool PK = sizeof(Real) == 4;
    const Real g = (Real)Ap->g;
    const Two<Real> N = {Nx, Ny};
    Side<Real> o = Trace<P, Real>::get(tr, NS, own, gp, g);
    Side<Real> n = Trace<P, Real>::get(tr, NS, slot, MT<P>::NG - 1 - gp, g);
    if (WD && sizeof(Real) == 8) {  // a dry side's trace comes without them
        if (!wet) complete<Real>(o, g);
        if (!wn) complete<Real>(n, g);
    }
    Real F0;
    Two<Real> F12;
    llf_sides_spherical<PK, Real>(g, o, n, N, sp, is_in, F0, F12);
    if (WD && wet != wn) wd_fixup_spherical<PK, Real>(g, o, n, N, w, sp, wet, wn, F0, F12);
    return Val3<Real>{F0, F12.x, F12.y};
}

// The master tables in constant memory, for the loops that run rolled (uniform indexes); FP32 entries twice,
// as the operand of a packed instruction
template <typename Real>
struct CoefType {
    using type = Real;
};
template <>
struct CoefType<float> {
    using type = Two<float>;
};
template <typename Real>
using Coef = typename CoefType<Real>::type;
__host__ __device__ constexpr Two<float> as_coef(float c) { return {c, c}; }
__host__ __device__ constexpr double as_coef(double c) { return c; }
__device__ __forceinline__ Two<float> pair_of(Two<float> c) { return c; }
__device__ __forceinline__ Two<double> pair_of(double c) { return {c, c}; }

template <int P, typename Real>
struct StageTab {
    static constexpr int ND = MT<P>::ND, NQ = MT<P>::NQ, NG = MT<P>::NG;
    Coef<Real> phi[NQ][ND], m0[NQ][ND], m1[NQ][ND], pw[NQ][ND];
    Real psi[NQ][4];
    Coef<Real> fphi[3][NG][ND];
    Real gw[NG];
};
template <int P, typename Real>
constexpr StageTab<P, Real> make_stage_tab() {
    using T = StageTab<P, Real>;
    T t{};
    for (int q = 0; q < T::NQ; ++q) {
        for (int k = 0; k < T::ND; ++k) {
            t.phi[q][k] = as_coef((Real)MT<P>::phi(k * T::NQ + q));
            t.m0[q][k] = as_coef((Real)MT<P>::mz((0 * T::NQ + q) * T::ND + k));
            t.m1[q][k] = as_coef((Real)MT<P>::mz((1 * T::NQ + q) * T::ND + k));
            t.pw[q][k] = as_coef((Real)MT<P>::phiw(q * T::ND + k));
        }
        for (int n = 0; n < 3; ++n) t.psi[q][n] = (Real)MT<P>::psi(n * T::NQ + q);
    }
    for (int g = 0; g < T::NG; ++g) t.gw[g] = (Real)MT<P>::gw(g);
    for (int f = 0; f < 3; ++f)
        for (int g = 0; g < T::NG; ++g)
            for (int k = 0; k < T::ND; ++k) t.fphi[f][g][k] = as_coef((Real)MT<P>::fphi((f * T::ND + k) * T::NG + g));
    return t;
}
template <int P, typename Real>
__constant__ const StageTab<P, Real> stage_tab = make_stage_tab<P, Real>();

// whether mode k's entry counts at any point (0: phi, 1: m0, 2: m1, 3: pw, 4: fphi)
template <int P>
constexpr bool counts_any(int what, int k) {
    using M = MT<P>;
    if (what == 4) {
        for (int i = 0; i < 3 * M::NG; ++i)
            if (counts(M::fphi((i / M::NG * M::ND + k) * M::NG + i % M::NG))) return true;
        return false;
    }
    for (int q = 0; q < M::NQ; ++q)
        if (counts(what == 0   ? M::phi(k * M::NQ + q)
                   : what == 1 ? M::mz((0 * M::NQ + q) * M::ND + k)
                   : what == 2 ? M::mz((1 * M::NQ + q) * M::ND + k)
                               : M::phiw(q * M::ND + k)))
            return true;
    return false;
}

// shared-memory layout of the stage kernel; mh: halo and boundary faces of a tile
template <int P, typename Real>
struct Smem {
    static constexpr int ND = MT<P>::ND;
    static __host__ __device__ size_t al(size_t b) { return (b + 15) & ~size_t(15); }
    static __host__ __device__ int nslot(int tile, int mh) { return 3 * tile + mh; }
    static __host__ __device__ size_t off_wet(int tile, int mh) {
        return (size_t)16 * MT<P>::NG * Trace<P, Real>::NV * nslot(tile, mh);
    }
    // halo staging (FP32): the state and bathymetry modes of each halo face's element, copied asynchronously
    static constexpr bool staged = sizeof(Real) == 4;
    static __host__ __device__ size_t off_halo(int tile, int mh) { return off_wet(tile, mh) + al((size_t)nslot(tile, mh)); }
    static __host__ __device__ size_t off_hbath(int tile, int mh) {
        return off_halo(tile, mh) + al(sizeof(double) * (size_t)3 * ND * mh);
    }
    static __host__ __device__ size_t bytes(int tile, int mh) {
        return staged ? off_hbath(tile, mh) + al(sizeof(Real) * (size_t)3 * mh) : off_halo(tile, mh);
    }
};

// asynchronous global -> shared copies of one 4- or 8-byte value (the thread does not wait for it)
template <typename Real>
__device__ __forceinline__ void cp_async_value(Real* dst, const Real* src) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(Real) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit_and_wait() {
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// resident CTAs per SM the register budget is sized for (p = 1 and p = 2 separately; tile 128, per 8 steps): p = 2 FP32 4
// (5 spills 592 B and runs 40 % slower), p = 1 FP32 5 (3-9 % faster than 4 on the bowl, tidal, levee and manufactured
// workloads; 6 spills and is slower), p = 2 FP64 3. p = 1 FP64: 4 without wetting/drying or analytic source (tidal channel
// of 524,288 0.94 against 1.11 ms with 3; one wave either way, 32,768, 0.154 against 0.155); 3 with the
// source (manufactured of 524,288 1.29 against 1.31 ms with 4, of 32,768 0.19 against 0.23; 4 wins where it saves the last
// wave, of 65,522 0.28 against 0.30); 3 with wetting/drying, which suits small meshes only (bowl of 8,192 0.193 against
// 0.206 ms, of 32,768 0.200 against 0.210, but of 131,072 0.34 against 0.33, of 524,288 1.01 against 0.91 and of 1,048,352
// 1.99 against 1.76): a budget by the number of waves is not built
#ifndef DGSW_F32_MB128
#define DGSW_F32_MB128 4
#endif
#ifndef DGSW_F64_MB128
#define DGSW_F64_MB128 3
#endif
#ifndef DGSW_F32_P1_MB128
#define DGSW_F32_P1_MB128 5
#endif
#ifndef DGSW_F64_P1_MB128
#define DGSW_F64_P1_MB128 4
#endif
#ifndef DGSW_F64_P1_FSRC_MB128
#define DGSW_F64_P1_FSRC_MB128 3
#endif
#ifndef DGSW_F64_P1_WD_MB128
#define DGSW_F64_P1_WD_MB128 3
#endif
// OCC = 1 selects the autotuner's alternative budget: one resident CTA fewer where the default holds
// several (more registers per thread), one more where it holds one (tile 256 in FP64)
template <int P, typename Real, int TILE, bool WD, bool FSRC, int OCC = 0>
struct MinBlocks {
    static constexpr int f32 = P == 1 ? DGSW_F32_P1_MB128 : DGSW_F32_MB128;
    static constexpr int f64 = P == 1 ? (WD ? DGSW_F64_P1_WD_MB128 : FSRC ? DGSW_F64_P1_FSRC_MB128 : DGSW_F64_P1_MB128)
                                      : DGSW_F64_MB128;
    static constexpr int base = sizeof(Real) == 4 ? (TILE == 128 ? f32 : 2) : (TILE == 128 ? f64 : 1);
    static constexpr int value = OCC == 0 ? base : (base > 1 ? base - 1 : base + 1);
};

// shared-memory capacity; with CAPPED the stride of the trace vectors is this compile-time constant, so every
// shared-memory access has an immediate offset. On quad meshes whose sides are powers of two a tile of 128 has 35 halo
// and boundary faces on average and 56 at most; with other sides (the Morton order cuts them into less compact tiles)
// 57 and 86, and those run with strides read at run time
template <int TILE>
struct TileCap {
    static constexpr int halo = TILE / 2;
};

// the barrier between traces and faces: warps arrive with their traces written and wait after the volume integral
__device__ __forceinline__ void stage_bar_init(unsigned long long* bar, unsigned warps) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)), "r"(warps)
                 : "memory");
}
__device__ __forceinline__ void stage_bar_arrive(unsigned long long* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(
                         (unsigned)__cvta_generic_to_shared(bar))
                     : "memory");
}
// polls of the bounded wait, about 4 us each: a second. All warps of a CTA arrive, so that a wait that runs out means a
// fault of this code
constexpr unsigned STAGE_BAR_POLLS = 1u << 18;
// false, and recorded in the status by whichever thread it happens to, when the wait runs out: its element's results
// stay unwritten, whatever the other warps' waits do
__device__ __forceinline__ bool stage_bar_wait(unsigned long long* bar, DevStatus* status,
                                               unsigned polls = STAGE_BAR_POLLS) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    for (unsigned i = 0; i < polls; ++i) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a)
            : "memory");
        if (done) return true;
    }
    atomicOr(&status->wait_failed, 1u);
    return false;
}

template <int P, typename Real, bool WD, bool FSRC, bool FRIC, int TILE, bool CAPPED, int OCC = 0, bool SPLIT = false>
__global__ void __launch_bounds__(TILE, (MinBlocks<P, Real, TILE, WD, FSRC, OCC>::value))
    rkdg_stage_kernel(const __grid_constant__ StageArgs<Real> A, int max_halo_rt) {
    static_assert(!SPLIT || (!WD && sizeof(Real) == 4), "stage increments: FP32 arithmetic without wetting/drying");
    const int max_halo = CAPPED ? TileCap<TILE>::halo : max_halo_rt;
    constexpr int ND = MT<P>::ND, NQ = MT<P>::NQ, NG = MT<P>::NG;
    using SM = Smem<P, Real>;
    using TR = Trace<P, Real>;
    const int NS = SM::nslot(TILE, max_halo);  // trace slots: 3 per tile element, then halo and boundary faces
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* tr = smem_raw;
    unsigned char* swet = smem_raw + SM::off_wet(TILE, max_halo);                         // [NS]
    double* shq = reinterpret_cast<double*>(smem_raw + SM::off_halo(TILE, max_halo));     // [3*ND][max_halo]
    Real* shb = reinterpret_cast<Real*>(smem_raw + SM::off_hbath(TILE, max_halo));        // [3][max_halo]
    __shared__ unsigned long long bar;

    // odd stages walk the tiles backwards: they start on the tiles the previous stage wrote last,
    // whose states are still in L2 (tiles are independent, so the results do not change)
    if ((int)blockIdx.x >= A.ntiles) {
        form_step_time(&A.time, (int)blockIdx.x - A.ntiles);
        return;
    }
    const int tile = A.reverse ? A.ntiles - 1 - (int)blockIdx.x : (int)blockIdx.x;
    const int e0 = tile * TILE;
    const int nloc = min(TILE, A.ne - e0);
    const int tid = threadIdx.x;
    const int d = e0 + tid;
    const bool active = tid < nloc;
    const int P_ = A.ne_pad;
    const Real g = (Real)A.g;
    const double* __restrict__ qs = A.qk[A.nterms - 1];  // this stage's state
    // the stage's time factors (ESSPRKStepper::GetTimeAtCurrentStage), formed during the previous step
    const StageTime& ST = A.clock->at[A.stage_index];
    const dgsw_fn_time& FT = ST.ft;
    // the face traces' basis values at the edge Gauss points, [face][mode][gp], for the halo traces. Measured per
    // step against compile-time tables per face (bit-identical results): FP32 at p = 2 -0.6 to -0.9 %; FP64 at
    // p = 2 -0.6 to +0.5 %, p = 1 +1 to +4 % (the shared-memory loads cost more than the divergence there), so
    // only FP32 at p = 2 uses it
    constexpr bool rt_face = P == 2 && sizeof(Real) == 4;
    // packed FP32 instructions (Two) throughout the FP32 kernels
    constexpr bool PK = sizeof(Real) == 4;
    __shared__ Real sfphi[rt_face ? 3 * ND * NG : 1];
    if (tid == 0) stage_bar_init(&bar, TILE / 32);
    if (rt_face && tid < 3 * ND * NG) {
        Real c = Real(0);
        sfor<0, 3 * ND * NG>([&](auto I) {
            constexpr int i = decltype(I)::value;
            if (tid == i) c = (Real)MT<P>::fphi(i);
        });
        sfphi[tid] = c;
    }
    __syncthreads();
    // the manufactured sine set's source inline, in both precisions; other sets go through fn_eval_dev
    const bool sine_set = FSRC && A.fn_set == DGSW_FN_MANUFACTURED_SINE;
    SineSrc<Real> SS;
    if (sine_set) SS = sine_src_load<Real>(ST);

    Real rhs[3][ND];
#pragma unroll
    for (int v = 0; v < 3; ++v)
#pragma unroll
        for (int k = 0; k < ND; ++k) rhs[v][k] = Real(0);
    // rhs += G c with (qx, qy) as one pair
    auto add_to = [&](int k, Real g0, Two<Real> g12, Two<Real> c) {
        const Two<Real> r = fma2<PK, Real>(g12, c, Two<Real>{rhs[1][k], rhs[2][k]});
        rhs[1][k] = r.x, rhs[2][k] = r.y;
        rhs[0][k] = fma_rn(g0, c.x, rhs[0][k]);
    };
    auto both = [](double c) { return Two<Real>{(Real)c, (Real)c}; };
    const StageTab<P, Real>& TB = stage_tab<P, Real>;
    // Rolled loops over the quadrature points (ROLL_V) and the faces (ROLL_F), their table entries read from
    // constant memory; unrolled, every entry is an immediate or a constant operand and zero entries are skipped. The
    // unrolled p = 2 and FP64 kernels outgrow the instruction caches (3.3 stalls on instruction fetch per issue at
    // FP64 p = 2). Measured per 8 steps of 524,288 triangles, unrolled -> rolled: FP64 p = 2 5.08 -> 4.53 ms (points)
    // -> 4.34 ms (points and faces), FP64 p = 1 manufactured 1.41 -> 1.36 ms, the FP64 bowl of 980,000 3.34 -> 3.25 ms;
    // FP32 p = 2 faces 2.08 -> 2.05 ms, points 2.08 -> 2.22 ms; FP32 p = 1 manufactured, points and faces,
    // 0.735 -> 0.749 ms; FP64 p = 1 channel 0.96 -> 1.00 ms or more; FP64 p = 2 without a source, closed basin 3.38 ->
    // 3.29 and channel 3.90 -> 3.60 ms (all with FP64's halo elements staged in shared memory, see below). So the FP32 points and all of FP32 p = 1 stay
    // unrolled, and FP64 p = 1 without source and wetting/drying.
    constexpr bool ROLL_V = sizeof(Real) == 8 && (P == 2 || FSRC || WD);
    constexpr bool ROLL_F = P == 2 || (sizeof(Real) == 8 && (FSRC || WD));
    // stage increments: the combination's increment terms sum_k a_k d_k + dt b_k sol_k in Real, loaded ahead of
    // the face loop
    Real dcomb[3][ND];
    auto split_comb = [&]() {
#pragma unroll
        for (int v = 0; v < 3; ++v)
#pragma unroll
            for (int k = 0; k < ND; ++k) dcomb[v][k] = Real(0);
        for (int j = 0; j < A.nterms; ++j) {
            const Real* __restrict__ dj = A.dk[j];
            if (dj) {
                const Real aj = (Real)A.a[j];
                Real t[3][ND];
#pragma unroll
                for (int v = 0; v < 3; ++v)
#pragma unroll
                    for (int k = 0; k < ND; ++k) t[v][k] = dj[(v * ND + k) * P_ + d];
                if constexpr (PK) {
#pragma unroll
                    for (int k = 0; k < ND; ++k) {
                        const Two<Real> r = fma2<PK, Real>(Two<Real>{t[1][k], t[2][k]}, aj, Two<Real>{dcomb[1][k], dcomb[2][k]});
                        dcomb[1][k] = r.x, dcomb[2][k] = r.y;
                        dcomb[0][k] = fma_rn(t[0][k], aj, dcomb[0][k]);
                    }
                } else {
#pragma unroll
                    for (int v = 0; v < 3; ++v)
#pragma unroll
                        for (int k = 0; k < ND; ++k) dcomb[v][k] += aj * t[v][k];
                }
            }
            if (j < A.nterms - 1 && A.bdt[j] != 0.0) {
                const Real* __restrict__ sj = A.dsolk[j];
                const Real bj = (Real)A.bdt[j];
                Real u[3][ND];
#pragma unroll
                for (int v = 0; v < 3; ++v)
#pragma unroll
                    for (int k = 0; k < ND; ++k) u[v][k] = sj[(v * ND + k) * P_ + d];
                if constexpr (PK) {
#pragma unroll
                    for (int k = 0; k < ND; ++k) {
                        const Two<Real> r = fma2<PK, Real>(Two<Real>{u[1][k], u[2][k]}, bj, Two<Real>{dcomb[1][k], dcomb[2][k]});
                        dcomb[1][k] = r.x, dcomb[2][k] = r.y;
                        dcomb[0][k] = fma_rn(u[0][k], bj, dcomb[0][k]);
                    }
                } else {
#pragma unroll
                    for (int v = 0; v < 3; ++v)
#pragma unroll
                        for (int k = 0; k < ND; ++k) dcomb[v][k] += bj * u[v][k];
                }
            }
        }
    };
    bool wet = false;
    // FP32 with capped tiles (at most TILE / 2 halo and boundary faces): thread h < nh owns halo face h, its record is
    // loaded now and its element's data copied asynchronously into shared memory while the own traces are formed.
    // FP64 loads the halo elements after its own traces, in every tile: the staging area, 6 KB (p = 1) or 11 KB (p = 2) a
    // CTA, put the resident CTAs' shared memory above 196 KB, which leaves the L1 28 KB for 512 or 384 threads' loads in
    // flight instead of 60. Measured per 8 steps of 524,288 triangles, with staging -> without: p = 1 closed basin 1.17 ->
    // 0.84 ms, channel 1.25 -> 0.97, bowl 1.03 -> 1.02; p = 2 closed basin 3.29 -> 2.68 ms, channel 3.60 -> 2.95,
    // manufactured 4.15 -> 3.54, bowl 2.91 -> 2.43. (Staged in the halo face's own trace slot, which takes no memory, p = 1
    // 0.92 ms; tiles sized to the mesh run 10 to 15 % slower with copies than with loads.)
    constexpr bool ASYNC = CAPPED && SM::staged;
    const int2 ti = A.tiles[tile];
    const int hoff = ti.x, nh = ti.y;
    // FP64: one thread asks L2 for the rows this CTA reads only at its end, the RK combination's earlier
    // stages, so that those loads start on L2 hits instead of HBM latency. Bulk prefetches want 16-byte aligned
    // ranges: state rows start on a multiple of TILE elements.
    if (sizeof(Real) == 8 && tid == 0) {
        auto prefetch = [](const void* p, unsigned bytes) {
            if (bytes >= 16)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes & ~15u) : "memory");
        };
        const unsigned rowb = (unsigned)((nloc + 1) & ~1) * 8u;
        for (int j = 0; j < A.nterms - 1; ++j) {
            for (int c = 0; c < 3 * ND; ++c) prefetch(A.qk[j] + (size_t)c * P_ + e0, rowb);
            if (A.bdt[j] != 0.0)
                for (int c = 0; c < 3 * ND; ++c) prefetch(A.solk[j] + (size_t)c * P_ + e0, rowb);
        }
    }
    // stage increments, last stage: the carried state's trailing part is read only in the epilogue; one
    // thread asks L2 for this tile's rows now, so that those loads start on L2 hits
    if constexpr (SPLIT) {
        if (A.last && tid == 0) {
            const unsigned rowb = (unsigned)((nloc + 3) & ~3) * 4u;
            for (int c = 0; c < 3 * ND; ++c)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(A.q0lo + (size_t)c * P_ + e0),
                             "r"(rowb)
                             : "memory");
        }
    }
    int2 hrec = make_int2(0, -1);
    if (ASYNC && tid < nh) hrec = A.halo[hoff + tid];
    bool hwet = false;
    // stage increments: the halo staging holds q0f in its first 3 ND Real rows and d_s in the next 3 ND
    // (the same bytes as 3 ND doubles)
    Real* shf = reinterpret_cast<Real*>(shq);
    auto issue_halo_copies = [&]() {
        if constexpr (SPLIT) {
#pragma unroll
            for (int c = 0; c < 3 * ND; ++c) cp_async_value<Real>(&shf[c * max_halo + tid], &A.q0f[c * P_ + hrec.x]);
            if (A.dk[A.nterms - 1]) {
#pragma unroll
                for (int c = 0; c < 3 * ND; ++c)
                    cp_async_value<Real>(&shf[(3 * ND + c) * max_halo + tid], &A.dk[A.nterms - 1][c * P_ + hrec.x]);
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3 * ND; ++c) cp_async_value<double>(&shq[c * max_halo + tid], &qs[c * P_ + hrec.x]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) cp_async_value<Real>(&shb[k * max_halo + tid], &A.bath[k * P_ + hrec.x]);
        hwet = A.wet_in[hrec.x] != 0;
    };
    // an element's stage state in Real: q_s (FP64 stage states) or q0f + d_s (stage increments)
    auto load_state = [&](Real (&q)[3][ND], int e) {
        if constexpr (SPLIT) {
            const Real* __restrict__ ds = A.dk[A.nterms - 1];
            if (ds) {
                Real a[3 * ND], b[3 * ND];
#pragma unroll
                for (int c = 0; c < 3 * ND; ++c) a[c] = A.q0f[c * P_ + e];
#pragma unroll
                for (int c = 0; c < 3 * ND; ++c) b[c] = ds[c * P_ + e];
#pragma unroll
                for (int c = 0; c < 3 * ND; ++c) q[c / ND][c % ND] = a[c] + b[c];
            } else {
#pragma unroll
                for (int c = 0; c < 3 * ND; ++c) q[c / ND][c % ND] = A.q0f[c * P_ + e];
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3 * ND; ++c) q[c / ND][c % ND] = (Real)qs[c * P_ + e];
        }
    };

    // ---------------- traces ----------------
    Real q[3][ND], b[3];
    Real Ji00 = Real(0), Ji01 = Real(0), Ji10 = Real(0), Ji11 = Real(0);
    Real x0 = 0, y0 = 0, x1 = 0, y1 = 0, x2 = 0, y2 = 0;
    // the vertex coordinates (analytic source). FP64 at p = 2, whose register budget is tightest, loads them after the
    // traces
    constexpr bool xy_early = sizeof(Real) == 4 || P == 1;
    auto load_xy = [&]() {
        if (FSRC) {
            const int n0 = A.enodes[d], n1 = A.enodes[P_ + d], n2 = A.enodes[2 * P_ + d];
            const double2 p0 = A.xy[n0], p1 = A.xy[n1], p2 = A.xy[n2];
            x0 = (Real)p0.x, y0 = (Real)p0.y, x1 = (Real)p1.x, y1 = (Real)p1.y, x2 = (Real)p2.x, y2 = (Real)p2.y;
        }
    };
    // the faces' weights too, where the register budget holds them across the volume integral
    constexpr bool fw_early = sizeof(Real) == 4 || P == 1;
    int meta[3];
    Real fw[3];
    if (active) {
        load_state(q, d);
        if (ASYNC && hrec.y >= 0) issue_halo_copies();
#pragma unroll
        for (int k = 0; k < 3; ++k) b[k] = A.bath[k * P_ + d];
        wet = A.wet_in[d] != 0;
#pragma unroll
        for (int f = 0; f < 3; ++f) meta[f] = A.fmeta[f * P_ + d];
        if constexpr (fw_early) {
#pragma unroll
            for (int f = 0; f < 3; ++f) fw[f] = A.fw[f * P_ + d];
        }
        Ji00 = A.geo[d], Ji01 = A.geo[P_ + d], Ji10 = A.geo[2 * P_ + d], Ji11 = A.geo[3 * P_ + d];
        if constexpr (xy_early) load_xy();
        // the three faces (needed also when dry: a wet neighbour evaluates the interface)
        sfor<0, 3>([&](auto FF) {
            constexpr int f = decltype(FF)::value;
            put_face<P, f, PK, Real>(tr, NS, 3 * tid + f, q, b, g, !WD || wet);
            swet[3 * tid + f] = wet ? 1 : 0;
        });
        // boundary faces: their ghost states. A dry element's has no flux. One call site for the three faces, as few
        // elements have such a face and almost none two; at p = 1 FP32 and plain FP64, whose registers are tightest, keep
        // three (with the loop FP32 spills: manufactured of 1,048,352, 8 steps, 1.36 against 1.22 ms; FP64 closed basin of
        // 1,048,352 1.79 against 1.67, of 2,048 0.130 against 0.118). Boundary-heavy FP64 meshes, 8 steps: 8,000 wet/dry
        // members of 18 triangles 0.50 -> 0.42 ms, 1,000 of 200 0.60 -> 0.52, with this, the one division and the kept 1 / h.
        auto ghost = [&](auto FF, int m, Real w) {
            const auto fc = FF;
            const int f = fc;
            const int kind = m & 7, slot = m >> 4;
            swet[slot] = wet ? 1 : 0;
            if (WD && !wet) return;
            const Two<Real> N = scaled_normal<Real>(f, Ji00, Ji01, Ji10, Ji11);
            ghost_face<P, Real>(&A, tr, NS, 3 * tid + f, slot, d, f, kind, A.halo[hoff + slot - 3 * TILE].x, N.x, N.y, w);
        };
        if constexpr (P == 2 || (sizeof(Real) == 8 && (WD || FSRC))) {
            int bnd = 0;
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                const int kind = meta[f] & 7;
                bnd |= (kind >= 1 && kind <= 4 ? 1 : 0) << f;
            }
            while (bnd) {
                const int f = __ffs(bnd) - 1;
                bnd &= bnd - 1;
                ghost(f, f == 0 ? meta[0] : (f == 1 ? meta[1] : meta[2]),
                      !fw_early ? A.fw[f * P_ + d] : f == 0 ? fw[0] : (f == 1 ? fw[1] : fw[2]));
            }
        } else {
            sfor<0, 3>([&](auto FF) {
                constexpr int f = decltype(FF)::value;
                const int kind = meta[f] & 7;
                if (kind >= 1 && kind <= 4) ghost(FF, meta[f], fw_early ? fw[f] : A.fw[f * P_ + d]);
            });
        }
    }
    // halo faces: faces of elements in other tiles across this tile's edges
    auto halo_trace = [&](int h, int face, const Real (&qh)[3][ND], const Real (&bh)[3], bool w) {
        const int slot = 3 * TILE + h;
        if constexpr (rt_face) {
            put_face_rt<P, PK, Real>(tr, NS, slot, qh, bh, sfphi + face * ND * NG, g);
        } else if (face == 0) {
            put_face<P, 0, PK, Real>(tr, NS, slot, qh, bh, g, !WD || w);
        } else if (face == 1) {
            put_face<P, 1, PK, Real>(tr, NS, slot, qh, bh, g, !WD || w);
        } else {
            put_face<P, 2, PK, Real>(tr, NS, slot, qh, bh, g, !WD || w);
        }
        swet[slot] = w ? 1 : 0;
    };
    if (ASYNC) {
        if (hrec.y >= 0) {
            if (!active) issue_halo_copies();  // threads past the last element of the last tile
            const int h = tid;
            cp_async_commit_and_wait();  // this thread's own copies
            Real qh[3][ND], bh[3];
            if constexpr (SPLIT) {
                if (A.dk[A.nterms - 1]) {
#pragma unroll
                    for (int c = 0; c < 3 * ND; ++c)
                        qh[c / ND][c % ND] = shf[c * max_halo + h] + shf[(3 * ND + c) * max_halo + h];
                } else {
#pragma unroll
                    for (int c = 0; c < 3 * ND; ++c) qh[c / ND][c % ND] = shf[c * max_halo + h];
                }
            } else {
#pragma unroll
                for (int c = 0; c < 3 * ND; ++c) qh[c / ND][c % ND] = (Real)shq[c * max_halo + h];
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) bh[k] = shb[k * max_halo + h];
            halo_trace(h, hrec.y, qh, bh, hwet);
        }
    } else {
#pragma unroll 1
        for (int h = tid; h < nh; h += TILE) {
            const int2 it = A.halo[hoff + h];
            Real qh[3][ND], bh[3];
            load_state(qh, it.x);
#pragma unroll
            for (int k = 0; k < 3; ++k) bh[k] = A.bath[k * P_ + it.x];
            halo_trace(h, it.y, qh, bh, A.wet_in[it.x] != 0);
        }
    }
    stage_bar_arrive(&bar);

    // ---------------- volume + source integrals ----------------
    if (active && wet) {
        if constexpr (!xy_early) load_xy();
        // bathymetry gradient: the projected bathymetry is linear, its gradient constant
        Real db0 = Real(0), db1 = Real(0);
        sfor<0, 3>([&](auto K) {
            constexpr int k = decltype(K)::value;
            constexpr double c0 = MT<P>::dphi((0 * ND + k) * NQ + 0);
            constexpr double c1 = MT<P>::dphi((1 * ND + k) * NQ + 0);
            if constexpr (counts(c0)) db0 += b[k] * (Real)c0;
            if constexpr (counts(c1)) db1 += b[k] * (Real)c1;
        });
        const Two<Real> gdb = {g * (db0 * Ji00 + db1 * Ji10), g * (db0 * Ji01 + db1 * Ji11)};
        auto volume_point = [&](auto GP) {
            const auto gp = GP;  // IC<gp> (unrolled) or an int
            Two<Real> m = {Real(0), Real(0)}, zb = {Real(0), Real(0)};  // (qx, qy), (ze, b)
            sfor<0, ND>([&](auto K) {
                constexpr int k = decltype(K)::value;
                auto add = [&](Two<Real> c) {
                    m = fma2<PK, Real>(Two<Real>{q[1][k], q[2][k]}, c, m);
                    if constexpr (k < 3)
                        zb = fma2<PK, Real>(Two<Real>{q[0][k], b[k]}, c, zb);
                    else
                        zb.x = fma_rn(q[0][k], c.x, zb.x);
                };
                if constexpr (ROLL_V) {
                    if constexpr (counts_any<P>(0, k)) add(pair_of(TB.phi[gp][k]));
                } else {
                    constexpr double c = MT<P>::phi(k * NQ + decltype(GP)::value);
                    if constexpr (counts(c)) add(both(c));
                }
            });
            // physical flux (swe_flux.hpp:5-25) along the two master directions J^-1(z, :): with the contravariant
            // momentum U = J^-1(z, 0) qx + J^-1(z, 1) qy it is (U, q U / h + pe J^-1(z, :))
            const Real h = zb.x + zb.y;
            const Real ih = Real(1) / h;
            const Real pe = g * zb.x * (Real(0.5) * zb.x + zb.y);
            Real X0 = Ji00, X1 = Ji10;
            if (A.spherical) {
                const int i = gp;
                const Real sp = A.sph[(3 * NG + i) * P_ + d];
                X0 *= sp, X1 *= sp;
            }
            const Real U0 = X0 * m.x + Ji01 * m.y, U1 = X1 * m.x + Ji11 * m.y;
            const Two<Real> G0 = fma2<PK, Real>(m, U0 * ih, mul2<PK, Real>(Two<Real>{X0, Ji01}, pe));
            const Two<Real> G1 = fma2<PK, Real>(m, U1 * ih, mul2<PK, Real>(Two<Real>{X1, Ji11}, pe));
            // bathymetry-slope source, swe_source.hpp:15-21 (the analytic source follows in its own loop,
            // except the manufactured sine set in FP32, added here: its sum then shares the phi w products)
            Real S0 = Real(0);
            Two<Real> S12 = mul2<PK, Real>(gdb, zb.x);
            if constexpr (FSRC && sizeof(Real) == 4) {
                if (sine_set) {
                    Real s0, s1, s2;
                    if constexpr (ROLL_V) {
                        s0 = TB.psi[gp][0], s1 = TB.psi[gp][1], s2 = TB.psi[gp][2];
                    } else {
                        constexpr int i = decltype(GP)::value;
                        s0 = (Real)MT<P>::psi(0 * NQ + i), s1 = (Real)MT<P>::psi(1 * NQ + i), s2 = (Real)MT<P>::psi(2 * NQ + i);
                    }
                    const Real xg = (Real)x0 * s0 + (Real)x1 * s1 + (Real)x2 * s2;
                    const Real yg = (Real)y0 * s0 + (Real)y1 * s1 + (Real)y2 * s2;
                    Two<Real> fs;
                    sine_src_eval<PK, Real>(SS, xg, yg, S0, fs);
                    S12 = add2<PK, Real>(S12, fs);
                }
            }
            // bottom friction, swe_source.hpp:29-51: S(qx, qy) -= Cf |u| / h (qx, qy), Cf the Chezy coefficient
            // or, for Manning, max(g n^2 / h^(1/3), Cf); |u| / h as sqrt(qx^2 + qy^2) / h^2 where the reference has
            // hypot of the velocities (within a few ulps; momenta are far from hypot's overflow range)
            if (FRIC) {
                const Real cf = A.friction == DGSW_FRICTION_MANNING ? manning_cf<Real>(A.manning[d], h, (Real)A.friction_cf)
                                                                    : (Real)A.friction_cf;
                const Real tau = cf * sqrt(m.x * m.x + m.y * m.y) * (ih * ih);
                S12 = fma2<PK, Real>(m, -tau, S12);
            }
            // int F . grad(phi) = sum_gp sum_z F . J^-1(z, :) dphi_z w
            sfor<0, ND>([&](auto K) {
                constexpr int k = decltype(K)::value;
                auto slope = [&](Two<Real> c) {  // the source, whose continuity part only an analytic source has
                    if constexpr (FSRC) {
                        add_to(k, S0, S12, c);
                    } else {
                        const Two<Real> r = fma2<PK, Real>(S12, c, Two<Real>{rhs[1][k], rhs[2][k]});
                        rhs[1][k] = r.x, rhs[2][k] = r.y;
                    }
                };
                if constexpr (ROLL_V) {
                    if constexpr (counts_any<P>(1, k)) add_to(k, U0, G0, pair_of(TB.m0[gp][k]));
                    if constexpr (counts_any<P>(2, k)) add_to(k, U1, G1, pair_of(TB.m1[gp][k]));
                    if constexpr (counts_any<P>(3, k)) slope(pair_of(TB.pw[gp][k]));
                } else {
                    constexpr int i = decltype(GP)::value;
                    constexpr double m0 = MT<P>::mz((0 * NQ + i) * ND + k);
                    constexpr double m1 = MT<P>::mz((1 * NQ + i) * ND + k);
                    constexpr double pw = MT<P>::phiw(i * ND + k);
                    if constexpr (counts(m0)) add_to(k, U0, G0, both(m0));
                    if constexpr (counts(m1)) add_to(k, U1, G1, both(m1));
                    if constexpr (counts(pw)) slope(both(pw));
                }
            });
        };
        if constexpr (ROLL_V) {
#pragma unroll 1
            for (int gp = 0; gp < NQ; ++gp) volume_point(gp);
        } else {
            sfor<0, NQ>(volume_point);
        }
        // analytic source_q(t, x_gp) (swe_source.hpp:9-14), in a loop of its own so that its temporaries are not
        // live together with the flux computation's
        // The manufactured sine set in FP64 on elements small against its wavelength (k times the
        // largest vertex offset from the centroid <= 0.05): sin and cos once at the centroid, turned to
        // each quadrature point by rotate_small; the point's offset from the centroid is
        // sum_i (psi_i - 1/3) (x_i - x_0), its coordinate never formed. Measured on 524,288 triangles at
        // p = 2: FP64 stage 212 -> 201 us; in FP32 the hardware sine/cosine per point stays cheaper
        // (114 against 116 us).
        const double xc = (x0 + x1 + x2) * (1.0 / 3.0), yc = (y0 + y1 + y2) * (1.0 / 3.0);
        bool near = false;
        if constexpr (sizeof(Real) == 8)
            near = sine_set && (double)SS.k * fmax(fmax(fmax(fabs(x0 - xc), fabs(x1 - xc)), fabs(x2 - xc)),
                                                     fmax(fmax(fabs(y0 - yc), fabs(y1 - yc)), fabs(y2 - yc))) <= 0.05;
        if constexpr (sizeof(Real) == 8) {
            if (FSRC && near) {
                double sxc, cxc, syc, cyc;
                sine_src_sincos<Real>(SS, xc, sxc, cxc);
                sine_src_sincos<Real>(SS, yc, syc, cyc);
                const double ex1 = x1 - x0, ex2 = x2 - x0, ey1 = y1 - y0, ey2 = y2 - y0;
                auto near_point = [&](auto GP) {
                    const auto gp = GP;
                    const int i = gp;
                    const double a1 = TB.psi[i][1] - 1.0 / 3.0, a2 = TB.psi[i][2] - 1.0 / 3.0;
                    double sx, cx, sy, cy;
                    rotate_small(sxc, cxc, SS.k * (ex1 * a1 + ex2 * a2), sx, cx);
                    rotate_small(syc, cyc, SS.k * (ey1 * a1 + ey2 * a2), sy, cy);
                    Real f0;
                    Two<Real> f12;
                    sine_src_terms<PK, Real>(SS, sx, cx, sy, cy, f0, f12);
                    sfor<0, ND>([&](auto K) {
                        constexpr int k = decltype(K)::value;
                        if constexpr (ROLL_V) {
                            if constexpr (counts_any<P>(3, k)) add_to(k, f0, f12, pair_of(TB.pw[gp][k]));
                        } else {
                            constexpr double pw = MT<P>::phiw(decltype(GP)::value * ND + k);
                            if constexpr (counts(pw)) add_to(k, f0, f12, both(pw));
                        }
                    });
                };
                if constexpr (ROLL_V) {
#pragma unroll 1
                    for (int gp = 0; gp < NQ; ++gp) near_point(gp);
                } else {
                    sfor<0, NQ>(near_point);
                }
            }
        }
        if (FSRC && !near && !(sizeof(Real) == 4 && sine_set)) {
            const Real xr0 = (Real)x0, xr1 = (Real)x1, xr2 = (Real)x2;
            const Real yr0 = (Real)y0, yr1 = (Real)y1, yr2 = (Real)y2;
#pragma unroll 1
            for (int gp = 0; gp < NQ; ++gp) {
                // FP32 path: Gauss-point coordinates in FP32 (the analytic source is evaluated in FP32)
                const Real xg = xr0 * TB.psi[gp][0] + xr1 * TB.psi[gp][1] + xr2 * TB.psi[gp][2];
                const Real yg = yr0 * TB.psi[gp][0] + yr1 * TB.psi[gp][1] + yr2 * TB.psi[gp][2];
                Val3<Real> r;
                if (sine_set)
                    // FP64 elements large against the wavelength: out of line, so that this rarely
                    // taken path keeps the kernel's hot code small
                    r = sine_src_far<Real>(&ST, xg, yg);
                else
                    r = fn_eval_dev<Real>(A.fn_set, A.fn_params, &FT, 1, xg, yg);
                sfor<0, ND>([&](auto K) {
                    constexpr int k = decltype(K)::value;
                    if constexpr (counts_any<P>(3, k)) add_to(k, r.v0, Two<Real>{r.v1, r.v2}, pair_of(TB.pw[gp][k]));
                });
            }
        }
        // the volume integrals stay in master-element units: sol = (|J| V + E) M^-1 / |J| is computed as
        // V M^-1 + (E / |J|) M^-1, with 1 / |J| in the faces' weights
    }
    double comb[3][ND];
    double bv[3] = {0.0, 0.0, 0.0};
    // the loads of the CTA's end: the RK combination's state terms and the wet/dry vertex depths, issued ahead
    // of the face loop
    auto load_end = [&]() {
        if constexpr (SPLIT) split_comb();
#pragma unroll
        for (int v = 0; v < 3; ++v)
#pragma unroll
            for (int k = 0; k < ND; ++k) comb[v][k] = 0.0;
        for (int j = 0; j < (SPLIT ? 0 : A.nterms); ++j) {
            const double* __restrict__ qj = A.qk[j];
            const double aj = A.a[j];
            double t[3][ND];
#pragma unroll
            for (int v = 0; v < 3; ++v)
#pragma unroll
                for (int k = 0; k < ND; ++k) t[v][k] = qj[(v * ND + k) * P_ + d];
            if (j < A.nterms - 1 && A.bdt[j] != 0.0) {
                const double* __restrict__ sj = A.solk[j];
                const double bj = A.bdt[j];
                double u[3][ND];
#pragma unroll
                for (int v = 0; v < 3; ++v)
#pragma unroll
                    for (int k = 0; k < ND; ++k) u[v][k] = sj[(v * ND + k) * P_ + d];
#pragma unroll
                for (int v = 0; v < 3; ++v)
#pragma unroll
                    for (int k = 0; k < ND; ++k) comb[v][k] += bj * u[v][k];
            }
#pragma unroll
            for (int v = 0; v < 3; ++v)
#pragma unroll
                for (int k = 0; k < ND; ++k) comb[v][k] += aj * t[v][k];
        }
        // wetting/drying: the element's vertex depths, loaded now (two dependent loads) so that their latency
        // overlaps the face loop instead of opening the wet/dry pass
        if (WD) {
            const int n0 = A.enodes[d], n1 = A.enodes[P_ + d], n2 = A.enodes[2 * P_ + d];
            bv[0] = A.nz[n0], bv[1] = A.nz[n1], bv[2] = A.nz[n2];
        }
    };
    if (!stage_bar_wait(&bar, A.status)) return;
    if (!active) return;

    // ---------------- face fluxes and lift, M^-1, RK combination, wet/dry ----------------
    // the RK combination's state terms, sum_j a_j q_j + dt b_j sol_j over the earlier stages plus
    // a_s q_s, in FP64: all loads of one term are issued together here so that their latency overlaps
    // the face loop below (one dependent load per value at the end of the CTA cost a global-memory
    // latency per value, per wave)
    if constexpr (!fw_early) {
#pragma unroll
        for (int f = 0; f < 3; ++f) fw[f] = A.fw[f * P_ + d];
    }
    load_end();
    // the faces' lift, rhs += T phi_k(gp) on face f
    auto lift = [&](auto FF, auto GP, Real T0, Two<Real> T12) {
        const auto fc = FF;
        const auto gc = GP;
        const int f = fc, gp = gc;
        sfor<0, ND>([&](auto K) {
            constexpr int k = decltype(K)::value;
            if constexpr (std::is_same<decltype(FF), int>::value) {
                if constexpr (counts_any<P>(4, k)) add_to(k, T0, T12, pair_of(TB.fphi[f][gp][k]));
            } else {
                constexpr double c = MT<P>::fphi((decltype(FF)::value * ND + k) * NG + decltype(GP)::value);
                if constexpr (counts(c)) add_to(k, T0, T12, both(c));
            }
        });
    };
    // on: a face between wet elements, or a boundary face of one; these run without branches, so that one face's
    // loads overlap another's arithmetic. special: an interface with one dry side, a levee, the spherical correction;
    // few elements have one of the first two, and a rolled loop takes them afterwards.
    bool on[3];
    int special = 0;
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        const int kind = meta[f] & 7;
        const bool wn = kind >= 5 ? wet : swet[meta[f] >> 4] != 0;
        const bool any = kind < 5 && (wet || wn);
        const bool sp = kind == 5 || (any && ((WD && wet != wn) || A.spherical));
        on[f] = any && !sp;
        if (sp) special |= 1 << f;
    }
    if (!A.spherical && (!WD || on[0] || on[1] || on[2])) {  // with the correction every face is special
        auto face = [&](auto FF) {
            const auto fc = FF;  // IC<f> (unrolled) or an int
            const int f = fc;
            const Two<Real> N = scaled_normal<Real>(f, Ji00, Ji01, Ji10, Ji11);
            const int m = f == 0 ? meta[0] : (f == 1 ? meta[1] : meta[2]);
            const Real w = f == 0 ? fw[0] : (f == 1 ? fw[1] : fw[2]);
            const bool o_f = f == 0 ? on[0] : (f == 1 ? on[1] : on[2]);
            const int slot = o_f ? m >> 4 : 3 * tid + f;  // a levee's payload is no slot
            sfor<0, NG>([&](auto GP) {
                constexpr int gp = decltype(GP)::value;
                const Side<Real> o = TR::get(tr, NS, 3 * tid + f, gp, g);
                const Side<Real> n = TR::get(tr, NS, slot, NG - 1 - gp, g);
                Real F0;
                Two<Real> F12;
                llf_sides<PK, Real>(g, o, n, N, w, F0, F12);
                // rhs -= F phi_k w |e|/2 / |J|; the flux's 1/2 is in the weight, |e|/2 / |J| in the flux
                const Real wg = (Real)(-0.5 * MT<P>::gw(gp));
                const Two<Real> T12 = mul2<PK, Real>(F12, wg);
                lift(FF, GP, o_f ? F0 * wg : Real(0), Two<Real>{o_f ? T12.x : Real(0), o_f ? T12.y : Real(0)});
            });
        };
        if constexpr (ROLL_F) {
#pragma unroll 1
            for (int f = 0; f < 3; ++f) face(f);
        } else {
            sfor<0, 3>(face);
        }
    }
    if (special) {
#pragma unroll 1
        for (int f = 0; f < 3; ++f) {
            if (!(special >> f & 1)) continue;
            const int fm = A.fmeta[f * P_ + d];
            const Real w = A.fw[f * P_ + d];
            const int kind = fm & 7;
            const bool is_in = fm & 8;
            if (kind == 5) {  // a levee interface's flux comes from levee.cu
                const double* Fl = A.levF + (size_t)(fm >> 4) * (6 * NG);
#pragma unroll 1
                for (int gp = 0; gp < NG; ++gp) {
                    const int at = is_in ? gp : 3 * NG + NG - 1 - gp;
                    const Real wg = -TB.gw[gp] * w;
                    lift(f, gp, (Real)Fl[at] * wg, Two<Real>{(Real)Fl[NG + at] * wg, (Real)Fl[2 * NG + at] * wg});
                }
                continue;
            }
            const int slot = fm >> 4;
            const bool wn = swet[slot] != 0;
            const Two<Real> N = scaled_normal<Real>(f, Ji00, Ji01, Ji10, Ji11);
            Real sp_next = A.spherical ? A.sph[f * NG * P_ + d] : Real(1);  // loaded a point ahead
#pragma unroll 1
            for (int gp = 0; gp < NG; ++gp) {
                Real F0;
                Two<Real> F12;
                if (A.spherical) {
                    const Real sp = sp_next;
                    if (gp + 1 < NG) sp_next = A.sph[(f * NG + gp + 1) * P_ + d];
                    const Val3<Real> r = spherical_point<P, WD, Real>(&A, tr, NS, 3 * tid + f, slot, gp, sp, is_in, wet, wn,
                                                                      N.x, N.y, w);
                    F0 = r.v0, F12 = {r.v1, r.v2};
                } else {
                    Side<Real> o = TR::get(tr, NS, 3 * tid + f, gp, g);
                    Side<Real> n = TR::get(tr, NS, slot, NG - 1 - gp, g);
                    if (WD && sizeof(Real) == 8) {  // a dry side's trace comes without them
                        if (!wet) complete<Real>(o, g);
                        if (!wn) complete<Real>(n, g);
                    }
                    llf_sides<PK, Real>(g, o, n, N, w, F0, F12);
                    wd_fixup<PK, Real>(g, o, n, N, w, wet, wn, F0, F12);
                }
                const Real wg = Real(-0.5) * TB.gw[gp];
                lift(f, gp, F0 * wg, mul2<PK, Real>(F12, wg));
            }
        }
    }
    // M^-1 (the diagonal master mass inverse; 1 / |J| is already in) and the SSP-RK stage combination
    const double bdt_s = A.bdt[A.nterms - 1];
    if constexpr (SPLIT) {
        const Real bs = (Real)bdt_s;
        // dn = dcomb + dt b_s (rhs M^-1), qx and qy packed (each lane the scalar mul and fma)
        Real (&dn)[3][ND] = dcomb;
        sfor<0, ND>([&](auto K) {
            constexpr int k = decltype(K)::value;
            const Real mk = (Real)MT<P>::minv(k);
            const Two<Real> s12 = mul2<PK, Real>(Two<Real>{rhs[1][k], rhs[2][k]}, mk);
            const Real sol[3] = {mul_rn(rhs[0][k], mk), s12.x, s12.y};
            if (A.store_sol) {
#pragma unroll
                for (int v = 0; v < 3; ++v) A.dsol_out[(v * ND + k) * P_ + d] = sol[v];
            }
            const Two<Real> r = fma2<PK, Real>(s12, bs, Two<Real>{dn[1][k], dn[2][k]});
            dn[1][k] = r.x, dn[2][k] = r.y;
            dn[0][k] = fma_rn(sol[0], bs, dn[0][k]);
        });
        bool has_nan = false;
        if (A.last) {
            // the new carried state q0f + q0lo + d_ns in FP64 (q0f + q0lo is exact there), split again into
            // its leading and trailing Real parts; q_0 is loaded here rather than with the increments (held
            // across the face loop its registers would spill; its leading part is an L1 or L2 hit from the
            // traces)
            Real hi[3][ND], lo[3][ND];
#pragma unroll
            for (int v = 0; v < 3; ++v)
#pragma unroll
                for (int k = 0; k < ND; ++k) {
                    hi[v][k] = A.q0f[(v * ND + k) * P_ + d];
                    lo[v][k] = A.q0lo[(v * ND + k) * P_ + d];
                }
#pragma unroll
            for (int v = 0; v < 3; ++v)
#pragma unroll
                for (int k = 0; k < ND; ++k) {
                    const int idx = (v * ND + k) * P_ + d;
                    const double qv = ((double)hi[v][k] + (double)lo[v][k]) + (double)dn[v][k];
                    has_nan |= isnan(qv);
                    const Real h2 = (Real)qv;
                    A.q0f_out[idx] = h2;
                    A.q0lo_out[idx] = (Real)(qv - (double)h2);
                }
        } else {
#pragma unroll
            for (int v = 0; v < 3; ++v)
#pragma unroll
                for (int k = 0; k < ND; ++k) {
                    has_nan |= isnan(dn[v][k]);
                    A.d_out[(v * ND + k) * P_ + d] = dn[v][k];
                }
        }
        A.wet_out[d] = wet ? 1 : 0;
        if (has_nan) {
            const unsigned long long counter = (unsigned long long)A.clock->step * A.nstages + A.stage_index;
            atomicOr(&A.status->nan_flag, 1u);
            atomicMin(&A.status->nan_key, (counter << 32) | (unsigned int)A.ref_of_dev[d]);
        }
        return;
    }
    double qn[3][ND];
    sfor<0, ND>([&](auto K) {
        constexpr int k = decltype(K)::value;
        const Real mk = (Real)MT<P>::minv(k);
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            const double sol = (double)(rhs[v][k] * mk);
            const int idx = (v * ND + k) * P_ + d;
            if (A.store_sol) A.sol_out[idx] = sol;
            qn[v][k] = comb[v][k] + bdt_s * sol;
        }
    });
    bool wet_new = wet;
    if (WD) {
        const double bmin = fmin(bv[0], fmin(bv[1], bv[2]));
        bool went_dry = false;
        wet_new = wetting_drying<ND, double>(qn, bv, bmin, A.h_o, A.h_o_thr, wet, went_dry);
        if (A.went_dry) A.went_dry[d] = went_dry ? 1 : 0;
    }
    bool has_nan = false;
#pragma unroll
    for (int v = 0; v < 3; ++v)
#pragma unroll
        for (int k = 0; k < ND; ++k) {
            has_nan |= isnan((double)qn[v][k]);
            A.q_out[(v * ND + k) * P_ + d] = qn[v][k];
        }
    A.wet_out[d] = wet_new ? 1 : 0;
    if (A.baryctr) {
        // slope_limiting_prepare_element_kernel (swe_CS_slope_limiter.hpp:9-20): vertex values through
        // T_basis_linear, barycentre value = vertex values . (1/3, 1/3, 1/3)
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            const double a = qn[v][0], b = qn[v][1], c = qn[v][2];
            const double l0 = a - b - c, l1 = a - b + c, l2 = a + 2.0 * b;
            A.baryctr[v * P_ + d] = l0 * (1.0 / 3.0) + l1 * (1.0 / 3.0) + l2 * (1.0 / 3.0);
        }
    }
    if (has_nan) {
        const unsigned long long counter = (unsigned long long)A.clock->step * A.nstages + A.stage_index;
        atomicOr(&A.status->nan_flag, 1u);
        atomicMin(&A.status->nan_key, (counter << 32) | (unsigned int)A.ref_of_dev[d]);
    }
}

// launchers, one translation unit per (order, precision, register budget); bit 3 of `mode` selects the
// alternative budget (OCC = 1)
constexpr int STAGE_MODE_OCC = 8;
// bit 4 of `mode`: the kernel with run-time shared-memory strides even where the mesh fits the caps
constexpr int STAGE_MODE_UNCAPPED = 16;
cudaError_t launch_stage_p1_f64(const StageArgs<double>& A, int tile, int ntiles, int max_halo,
                                int mode, cudaStream_t s);
cudaError_t launch_stage_p1_f32(const StageArgs<float>& A, int tile, int ntiles, int max_halo,
                                int mode, cudaStream_t s);
cudaError_t launch_stage_p2_f64(const StageArgs<double>& A, int tile, int ntiles, int max_halo,
                                int mode, cudaStream_t s);
cudaError_t launch_stage_p2_f32(const StageArgs<float>& A, int tile, int ntiles, int max_halo,
                                int mode, cudaStream_t s);
cudaError_t launch_stage_p1_f64_occ(const StageArgs<double>& A, int tile, int ntiles, int max_halo,
                                    int mode, cudaStream_t s);
cudaError_t launch_stage_p1_f32_occ(const StageArgs<float>& A, int tile, int ntiles, int max_halo,
                                    int mode, cudaStream_t s);
cudaError_t launch_stage_p2_f64_occ(const StageArgs<double>& A, int tile, int ntiles, int max_halo,
                                    int mode, cudaStream_t s);
cudaError_t launch_stage_p2_f32_occ(const StageArgs<float>& A, int tile, int ntiles, int max_halo,
                                    int mode, cudaStream_t s);
// stage increments (StageArgs::dk ...): the default budget, or the alternative one with bit 3 of `mode`
cudaError_t launch_stage_p1_f32_split(const StageArgs<float>& A, int tile, int ntiles, int max_halo,
                                      int mode, cudaStream_t s);
cudaError_t launch_stage_p2_f32_split(const StageArgs<float>& A, int tile, int ntiles, int max_halo,
                                      int mode, cudaStream_t s);

// whether every tile of a mesh fits the compile-time shared-memory capacity of the capped kernels
inline bool stage_fits_caps(int tile, int max_halo) {
    return max_halo <= (tile == 128 ? TileCap<128>::halo : TileCap<256>::halo);
}

// with `allow_capped` false the kernel with run-time strides runs even where the mesh fits the caps: its
// shared memory is sized to the mesh's largest tile, and with less shared memory per SM the L1 cache that
// shares its storage is larger (the autotuner times both)
template <int P, typename Real, bool WD, bool FSRC, bool FRIC, int TILE, int OCC, bool SPLIT = false>
cudaError_t launch_stage_impl(const StageArgs<Real>& A, int ntiles, int max_halo, bool allow_capped, cudaStream_t s) {
    const bool capped = allow_capped && max_halo <= TileCap<TILE>::halo;
    auto kern = capped ? rkdg_stage_kernel<P, Real, WD, FSRC, FRIC, TILE, true, OCC, SPLIT>
                       : rkdg_stage_kernel<P, Real, WD, FSRC, FRIC, TILE, false, OCC, SPLIT>;
    // the run-time-stride kernel loads its halo faces' elements straight from global memory, so its allocation ends
    // before the staging area
    const size_t smem = capped ? Smem<P, Real>::bytes(TILE, TileCap<TILE>::halo) : Smem<P, Real>::off_halo(TILE, max_halo);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)(ntiles + A.n_time), TILE, smem, s>>>(A, max_halo);
    return cudaGetLastError();
}

template <int P, typename Real, bool WD, bool FSRC, bool FRIC, int OCC, bool SPLIT = false>
cudaError_t launch_stage_tile(const StageArgs<Real>& A, int tile, int ntiles, int max_halo, int mode, cudaStream_t s) {
    const bool allow_capped = !(mode & STAGE_MODE_UNCAPPED);
    switch (tile) {
        case 128:
            return launch_stage_impl<P, Real, WD, FSRC, FRIC, 128, OCC, SPLIT>(A, ntiles, max_halo, allow_capped, s);
        case 256:
            return launch_stage_impl<P, Real, WD, FSRC, FRIC, 256, OCC, SPLIT>(A, ntiles, max_halo, allow_capped, s);
        default:
            return cudaErrorInvalidValue;
    }
}

// wetting/drying, function source and bottom friction select the instantiation (bit 0, 1, 2 of `mode`)
template <int P, typename Real, int OCC>
cudaError_t launch_stage_dispatch(const StageArgs<Real>& A, int tile, int ntiles, int max_halo,
                                  int mode, cudaStream_t s) {
    switch (mode & 7) {
        case 0: return launch_stage_tile<P, Real, false, false, false, OCC>(A, tile, ntiles, max_halo, mode, s);
        case 1: return launch_stage_tile<P, Real, true, false, false, OCC>(A, tile, ntiles, max_halo, mode, s);
        case 2: return launch_stage_tile<P, Real, false, true, false, OCC>(A, tile, ntiles, max_halo, mode, s);
        case 3: return launch_stage_tile<P, Real, true, true, false, OCC>(A, tile, ntiles, max_halo, mode, s);
        case 4: return launch_stage_tile<P, Real, false, false, true, OCC>(A, tile, ntiles, max_halo, mode, s);
        case 5: return launch_stage_tile<P, Real, true, false, true, OCC>(A, tile, ntiles, max_halo, mode, s);
        case 6: return launch_stage_tile<P, Real, false, true, true, OCC>(A, tile, ntiles, max_halo, mode, s);
        default: return launch_stage_tile<P, Real, true, true, true, OCC>(A, tile, ntiles, max_halo, mode, s);
    }
}

// the stage-increment kernels (FP32, no wetting/drying): function source and bottom friction select the
// instantiation (bits 1 and 2 of `mode`; bit 0, wetting/drying, must be clear)
template <int P, int OCC>
cudaError_t launch_stage_split_dispatch(const StageArgs<float>& A, int tile, int ntiles, int max_halo,
                                        int mode, cudaStream_t s) {
    switch (mode & 7) {
        case 0: return launch_stage_tile<P, float, false, false, false, OCC, true>(A, tile, ntiles, max_halo, mode, s);
        case 2: return launch_stage_tile<P, float, false, true, false, OCC, true>(A, tile, ntiles, max_halo, mode, s);
        case 4: return launch_stage_tile<P, float, false, false, true, OCC, true>(A, tile, ntiles, max_halo, mode, s);
        case 6: return launch_stage_tile<P, float, false, true, true, OCC, true>(A, tile, ntiles, max_halo, mode, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace dgsw

#endif
