// hs_mixed.cu -- mixed-precision batched HSolve step (sm_103a).
//
// A persistent kernel: each CTA owns a list of forests (groups of cells,
// hs_mixed.cuh) packed by size on the host and steps each forest for
// `nsteps` steps before moving on.  Per step, the whole CTA:
//   tick 0    stimulus schedule (a thread per cell)
//   assembly  every node in parallel: FP32 rate lookup and gate update for
//             each channel slot, conductances, the K(Ca) 2-D gate, SynChans;
//             FP64 matrix row into the elimination arrays
//   forward   levels deepest first, a barrier per level: pull the children's
//             eliminated rows, FP64 pivot reciprocal
//   backward  levels root first: VMid = g - f * VMid[parent] (FP64)
//   update    V = 2 VMid - V, Ca pools (FP32)
//   outputs   SpikeGens, trace samples (a thread per cell).
// stepForestWS overlaps assembly and forward elimination of a forest, stepPair
// the whole elimination of one with the assembly of another.
// The update and outputs of a step are done at the start of the next step's
// assembly (and after the last step), which saves a pass over the nodes.
// Reference routines: hsolve/HSolveActive.cpp:45-332, hsolve/HSolvePassive.cpp:
// 246-401 (the same elimination, tree form), biophysics/HHChannel2D.cpp:327-369,
// biophysics/SynChan.cpp:200-224, synapse/SimpleSynHandler.cpp:98-113,
// biophysics/SpikeGen.cpp:202-216.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "hs_exact.cuh"
#include "hs_mixed.cuh"
#include "hs_shared.h"

namespace hsg {


// Stop step of a cell (none unless the batch set some).
__device__ __forceinline__ unsigned long long stopOf(const MixBatch& b, uint32_t cell) {
    return b.anyStop ? b.stopStep[cell] : ~0ull;
}

// The batch's channel type `tj` (one 16-byte read-only load).
__device__ __forceinline__ ChanType chanType(const MixBatch& b, uint32_t tj) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(b.chanTypes + tj));
    ChanType t;
    *reinterpret_cast<uint4*>(&t) = v;
    return t;
}

// Reciprocal of a positive FP64 pivot: the hardware FP64 reciprocal
// estimate (rcp.approx.ftz.f64, relative error about 1e-6 measured over
// 1e-9..1e9) refined by one Newton-Raphson step x <- x + x(1 - d x), which
// squares the error (about 1e-12).
__device__ __forceinline__ double rcpPivot(double d) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
    const double e = fma(-d, x, 1.0);
    return fma(x, e, x);
}

// (float)x by integer operations (the conversion issues at the FP64 rate):
// round to nearest even in the float's normal range, the instruction outside.
__device__ __forceinline__ float narrowD(double x) {
    const unsigned long long b = (unsigned long long)bitsOf(x);
    const uint32_t h = (uint32_t)(b >> 32) & 0x7FFFFFFFu;
    if (h - 0x38100000u >= 0x0FD00000u) return (float)x;
    const uint32_t m = (uint32_t)((b & 0x7FFFFFFFFFFFFFFFull) >> 29) - 0x1C0000000ull, rest = (uint32_t)b & 0x1FFFFFFFu;
    const uint32_t up = rest + (m & 1u) > 0x10000000u ? 1u : 0u;
    return __uint_as_float((m + up) | ((uint32_t)(b >> 32) & 0x80000000u));
}

__device__ __forceinline__ float powi(float x, int p, float pf) {
    switch (p) {
    case 1: return x;
    case 2: return x * x;
    case 3: return x * x * x;
    case 4: { float y = x * x; return y * y; }
    default: return x > 0.f ? __powf(x, pf) : 0.f;
    }
}

struct RowF {
    const float* p;
    float frac;
};

__device__ __forceinline__ RowF rowF(const float* T, uint32_t nCol, uint32_t nRows, float x, float mn,
                                     float mx, float invDx) {
    x = fminf(fmaxf(x, mn), mx);
    float div = (x - mn) * invDx;
    unsigned int i = min((unsigned int)div, nRows - 2);   // rows i and i+1 exist
    RowF r;
    r.frac = div - (float)i;
    r.p = T + 2 * (size_t)i * nCol;
    return r;
}

// Exact widening of an FP32 value to FP64 with integer operations (the
// FP32-to-FP64 conversion instruction issues at the FP64 rate on this GPU,
// integer operations at the full rate).  IEEE binary32 -> binary64: sign
// kept, exponent rebiased by 1023 - 127 = 896, fraction shifted left by 29;
// zero and subnormal inputs give a signed zero, Inf/NaN stay Inf/NaN.
__device__ __forceinline__ double widenF(float x) {
    const uint32_t u = __float_as_uint(x);
    const uint32_t e = (u >> 23) & 0xFFu;
    const uint32_t sign = u & 0x80000000u;
    const uint32_t e64 = e == 0xFFu ? 0x7FFu : e + 896u;
    const uint32_t hi = e == 0 ? sign : (sign | (e64 << 20) | ((u >> 3) & 0xFFFFFu));
    const uint32_t lo = e == 0 ? 0u : (u << 29);
    return __hiloint2double((int)hi, (int)lo);
}

// Column `col` (A at col, B at col + 1) between the row and the next:
// {A, B, differences to the next row}, and their interpolation.
__device__ __forceinline__ float4 rowOf(const RowF& r, int col) {
    return __ldg(reinterpret_cast<const float4*>(r.p + 2 * col));
}
__device__ __forceinline__ float2 lerp(const float4& q, float frac) {
    return make_float2(fmaf(q.z, frac, q.x), fmaf(q.w, frac, q.y));
}
__device__ __forceinline__ float2 lookupF(const RowF& r, int col) { return lerp(rowOf(r, col), r.frac); }

// A gate state held as the unevaluated sum hi + lo of two FP32 numbers
// (|lo| <= ulp(hi)/2), about 48 significant bits.  Adding an FP32 increment
// uses Knuth's TwoSum (the exact rounding error of hi + d) and Dekker's
// Fast2Sum to renormalise, all on the FP32 pipe: a plain FP32 state would
// lose the small per-step increments of slow gates, and an FP64 add issues
// at 1/64 of the FP32 rate on this GPU, on the pipe the elimination needs.
__device__ __forceinline__ float2 addPair(float2 x, float d) {
    const float s = __fadd_rn(x.x, d);
    const float bv = __fsub_rn(s, x.x);
    const float err = __fadd_rn(__fsub_rn(x.x, __fsub_rn(s, bv)), __fsub_rn(d, bv));
    const float lo = __fadd_rn(x.y, err);
    const float hi = __fadd_rn(s, lo);
    return make_float2(hi, __fsub_rn(lo, __fsub_rn(hi, s)));
}

// New value of a gate with state x over one step, from C1, C2 of its table
// row.  The reference's trapezoidal step (x(2-T) + dt C1)/T with T = 1 + h,
// h = dt/2 C2 (hsolve/HSolveActive.cpp:272-273) is the same number as
// x + (dt C1 - 2 h x)/(1 + h): the increment is computed in FP32 and added
// to the two-float state.  Instantaneous gates: x = C1/C2.
__device__ __forceinline__ float2 gateStep(float2 C, float2 x, float dt, float hdt, bool inst) {
    if (inst) return make_float2(__fdividef(C.x, C.y), 0.f);
    const float h = hdt * C.y;
    return addPair(x, __fdividef(fmaf(-2.0f * h, x.x, dt * C.x), 1.0f + h));
}

__device__ __forceinline__ void interp2dF(const float* g2d, const C2dType& t, float x, float y, float& A, float& B) {
    const uint32_t nx = t.nx, ny = t.ny;
    const float* T = g2d + t.tab;
    x = fminf(fmaxf(x, t.xmin), t.xmax);
    y = fminf(fmaxf(y, t.ymin), t.ymax);
    float xv = (x - t.xmin) * t.invDx;
    float yv = (y - t.ymin) * t.invDy;
    uint32_t xi = min((uint32_t)xv, nx - 1), yi = min((uint32_t)yv, ny - 1);
    float xF = xv - (float)xi, yF = yv - (float)yi;
    bool endX = xi == nx - 1, endY = yi == ny - 1;
    const float* p00 = T + 2 * ((size_t)xi * ny + yi);
    const float2 z00 = __ldg(reinterpret_cast<const float2*>(p00));
    float2 z10 = make_float2(0.f, 0.f), z01 = z10, z11 = z10;
    if (!endX) z10 = __ldg(reinterpret_cast<const float2*>(p00 + 2 * ny));
    if (!endY) z01 = __ldg(reinterpret_cast<const float2*>(p00 + 2));
    if (!endX && !endY) z11 = __ldg(reinterpret_cast<const float2*>(p00 + 2 * ny + 2));
    float xFyF = xF * yF;
    float w00 = 1.f - xF - yF + xFyF, w10 = xF - xFyF, w01 = yF - xFyF;
    A = z00.x * w00 + z10.x * w10 + z01.x * w01 + z11.x * xFyF;
    B = z00.y * w00 + z10.y * w10 + z01.y * w01 + z11.y * xFyF;
}

// Dynamic shared memory of the stepping kernels: the prototypes, the words of
// the forests under way (ForestCtl), kWsLevels level counters, 4 words (the
// cluster's barrier), the level offsets, then the forest's arrays.
extern __shared__ __align__(16) unsigned char smem[];
__device__ __forceinline__ unsigned char* sTypes() { return smem; }
__device__ __forceinline__ uint32_t* sDone() { return reinterpret_cast<uint32_t*>(smem + kTypeBytes + kCtlBytes); }
__device__ __forceinline__ uint32_t* sBarrier() { return sDone() + kWsLevels; }
__device__ __forceinline__ uint32_t* sLevels() { return sBarrier() + 4; }
__device__ __forceinline__ double* sArea() { return reinterpret_cast<double*>(smem + kAreaBytes); }

// Of the forest a CTA steps, what its threads need now and then, kept here and
// not in their registers (64 a thread; see hsForestStepMixed).
struct ForestCtl {
    unsigned long long step;     // of the step under way
    uint32_t syn0, syn1;         // its SynChans
    uint32_t forest;
    MixForest F;
};
__device__ __forceinline__ volatile ForestCtl& sCtl(uint32_t g = 0) {
    return reinterpret_cast<volatile ForestCtl*>(sTypes() + kTypeBytes)[g];
}
static_assert(2 * sizeof(ForestCtl) <= kCtlBytes, "room for the forest's words");

// The batch's prototypes in shared memory.
__device__ __forceinline__ const ChanType* sChanTypes() { return reinterpret_cast<const ChanType*>(sTypes()); }
__device__ __forceinline__ const C2dType* sC2dTypes() { return reinterpret_cast<const C2dType*>(sChanTypes() + kMaxChanTypes); }
__device__ __forceinline__ const SynType* sSynTypes() { return reinterpret_cast<const SynType*>(sC2dTypes() + kMaxC2dTypes); }

// What a channel's X and Y gates read: their states and table rows.
struct ChanIn {
    float2 x, y;
    float4 rx, ry;
};

// One compartment node of the assembly: first the update left over from the
// previous step (V = 2 VMid - V, then the node's Ca pool; `update`), then
// channels, K(Ca), SynChans and the FP64 matrix row.
// Bound by the latency of a node's chain (~14,000 cycles on a lone cell, 7
// warps a sub-partition to hide it): the prototypes are in shared memory, a
// gate's table row is one 16-byte read, a channel's states and rows are read
// while the channel before it is computed and before its states are stored
// (a load does not pass a store it may alias), and of FP64 instructions, 76
// cycles each on this GPU, only the membrane's own five are left.
// kAhead: that reading ahead, for ~12 registers.  Without it in the kernels
// that hold several ways to step a forest, where it would spill.
template <bool kAhead>
__device__ __forceinline__ void assembleNode(const MixBatch& b, uint32_t n, uint32_t info, bool update,
                                             double vmPrev, double& diag, double& rhs) {
    const uint64_t ld = b.ld;
    const float dt = b.dtf, hdt = 0.5f * b.dtf;
    // ---- node data
    double V = b.V[n];
    const uint32_t types = __ldg(b.ctype4 + n);
    float2* const st = b.state + n;
    const bool pool = info & kNodePool;
    float ca = 0.f, c0v = 0.f, pg1 = 0.f, pf2 = 0.f, pbas = 0.f, pceil = 0.f, pfloor = 0.f, cgP = 0.f, cgeP = 0.f;
    if (pool) {
        ca = b.poolCa[n];
        if (update) {
            c0v = b.poolC[n];
            pg1 = __ldg(b.poolG1 + n);
            pf2 = __ldg(b.poolF2 + n);
            pbas = __ldg(b.poolBasal + n);
            pceil = __ldg(b.poolCeil + n);
            pfloor = __ldg(b.poolFloor + n);
            cgP = b.caG[n];
            cgeP = b.caGE[n];
        }
    }
    // ---- the previous step's update
    if (update) {
        const double Vold = V;
        V = fma(2.0, vmPrev, -Vold);
        b.V[n] = V;
        if (pool) {
            const float vca = narrowD(b.caAdvance == 1 ? vmPrev : Vold);
            const float act = fmaf(-cgP, vca, cgeP);
            // c f1 + f2 act with f1 = 1 - g1 (g1 = 1 - f1 from FP64)
            float c = fmaf(-pg1, c0v, c0v) + pf2 * act;
            float cav = pbas + c;
            if (pceil > 0.f && cav > pceil) { cav = pceil; c = cav - pbas; }
            if (cav < pfloor) { cav = pfloor; c = cav - pbas; }
            b.poolC[n] = c;
            b.poolCa[n] = cav;
            ca = cav;
        }
    }
    // ---- HHChannels: trapezoidal gates on the V (or Ca) table rows
    const float v = narrowD(V);
    const RowF vr = rowF(b.vTab, b.vCol, b.vRows, v, b.vMin, b.vMax, b.vInvDx);
    const uint32_t k2 = (info >> 8) & kNoK2;
    float G = 0.f, GE = 0.f, cg = 0.f, cge = 0.f;
#pragma unroll
    for (int j = 0; j < kMaxChan; ++j) {
        const uint32_t tj = (types >> (8 * j)) & 0xFF;
        if (tj == kNoType) break;       // channels fill the slots in order
        const ChanType t = sChanTypes()[tj];
        const float gb = __ldg(b.gbar + (uint64_t)j * ld + n);
        float2* const sj = st + (uint64_t)(3 * j) * ld;
        ChanIn in;
        auto readX = [&]() {
            in.x = sj[0];
            in.rx = rowOf(vr, t.colX);
        };
        auto readY = [&]() {
            in.y = sj[ld];
            in.ry = rowOf(vr, t.colY);
        };
        if (kAhead && t.xp) readX();
        if (kAhead && t.yp) readY();
        float frac = 1.f;
        if (t.xp) {
            if (!kAhead) readX();
            const float2 x = gateStep(lerp(in.rx, vr.frac), in.x, dt, hdt, t.instant & 1);
            sj[0] = x;
            frac *= powi(x.x, t.xp, t.xp < 0 ? __ldg(&b.chanPow[tj].x) : 0.f);
        }
        if (t.yp) {
            if (!kAhead) readY();
            const float2 y = gateStep(lerp(in.ry, vr.frac), in.y, dt, hdt, t.instant & 2);
            sj[ld] = y;
            frac *= powi(y.x, t.yp, t.yp < 0 ? __ldg(&b.chanPow[tj].y) : 0.f);
        }
        if (t.zp) {
            float2 C;
            if (t.zCa) C = lookupF(rowF(b.caTab, b.caCol, b.caRows, ca, b.caMin, b.caMax, b.caInvDx), t.colZ);
            else C = lookupF(vr, t.colZ);
            const float2 z = gateStep(C, sj[2 * ld], dt, hdt, t.instant & 4);
            sj[2 * ld] = z;
            frac *= powi(z.x, t.zp, t.zp < 0 ? __ldg(&b.chanPow[tj].z) : 0.f);
        }
        const float gk = gb * frac;
        G += gk;
        GE = fmaf(gk, t.ek, GE);
        if (t.caTarget) {
            cg += gk;
            cge = fmaf(gk, t.ek, cge);
        }
    }
    if (pool) {
        b.caG[n] = cg;
        b.caGE[n] = cge;
    }
    // ---- what the end of the chain needs
    const double hs2 = __ldg(b.HS2 + n), cmdt = __ldg(b.CmByDt + n), emrm = __ldg(b.EmByRm + n);
    uint32_t s0 = 0, s1 = 0;
    if (info & kNodeSyn) {
        s0 = __ldg(b.syn0 + n);
        s1 = __ldg(b.syn0 + n + 1);
    }
    // ---- HHChannel2D (K(Ca)) on this step's Vm and Ca
    if (k2 != kNoK2) {
        const C2dType& t = sC2dTypes()[k2];
        const float k2x = b.k2x[n], k2g = __ldg(b.k2gbar + n);
        const float x = t.dep0 == 0 ? v : t.dep0 == 1 ? ca : 0.f;
        const float y = t.dep1 == 0 ? v : t.dep1 == 1 ? ca : 0.f;
        float A, B;
        interp2dF(b.g2d, t, x, y, A, B);
        float X = k2x;
        if (t.instant & 1) X = __fdividef(A, B);
        else if (B > 1.0e-10f) {
            // HHChannelBase::integrate, X e + (A/B)(1 - e) with e = exp(-B dt),
            // as X + (A/B - X)(1 - e), 1 - e = -expm1(-B dt) (no cancellation)
            const float em = -expm1f(-B * dt);
            X = fmaf(__fdividef(A, B) - X, em, X);
        } else X = fmaf(A, dt, X);
        b.k2x[n] = X;
        const float gk = k2g * powi(X, t.xp, t.xpf);
        G += gk;
        GE = fmaf(gk, t.ek, GE);
    }
    // ---- SynChans: conductances of this step, advanced beforehand (synapseStep)
    for (uint32_t k = s0; k < s1; ++k) {
        const float2 g = b.synGk[k];
        G += g.x;
        GE += g.y;
    }
    diag = hs2 + widenF(G);
    rhs = fma(V, cmdt, emrm) + widenF(GE);
    if (info & kNodeInject) rhs += b.injVal[__ldg(b.injIdx + n)];
}

// SynChan k over step `step`: the events delivered (SimpleSynHandler, weight
// / dt each), the dual exponential X, Y, and the conductance Gk and Gk Ek
// the assembly of that step adds.  Needs no Vm, so it runs ahead of the
// assembly (see stepForest).
__device__ __forceinline__ void synapseStep(const MixBatch& b, uint32_t k, unsigned long long step) {
    if (step >= stopOf(b, __ldg(b.synCell + k))) return;
    const SynType& t = sSynTypes()[__ldg(b.synType + k)];
    uint32_t e = b.evCur[k];
    const uint32_t end = __ldg(b.evEnd + k);
    const float sx = b.synX[k], sy = b.synY[k], nm = __ldg(b.synNorm + k);
    float act = 0.f;
    while (e < end && __ldg(b.evStep + e) <= step) act += __ldg(b.evAct + e++);
    b.evCur[k] = e;
    const float X = fmaf(act, t.xc1, sx * t.xc2);
    const float Y = fmaf(X, t.yc1, sy * t.yc2);
    b.synX[k] = X;
    b.synY[k] = Y;
    const float gk = Y * nm;
    b.synGk[k] = make_float2(gk, gk * t.ek);
}

// Elimination arrays of a forest: pivots/couplings D, right-hand sides R,
// off-diagonals OFF, topology TOPO and PAR (forest-local indices).  As
// addresses computed from a word or two, not as pointers kept: the stepping
// kernels have 64 registers a thread, and a spilled pointer is an L2 access
// on the elimination's chain.
struct SharedRows {              // all of them, `cap` nodes, from the area's double `first`
    uint32_t cap, first;
    __device__ __forceinline__ double* base() const { return sArea() + first; }
    __device__ __forceinline__ double& D(uint32_t i) const { return base()[i]; }
    __device__ __forceinline__ double& R(uint32_t i) const { return base()[cap + i]; }
    __device__ __forceinline__ double* side(bool r) const { return base() + (r ? cap : 0); }     // R or D
    __device__ __forceinline__ double& OFF(uint32_t i) const { return base()[2 * cap + i]; }
    __device__ __forceinline__ uint32_t& TOPO(uint32_t i) const { return reinterpret_cast<uint32_t*>(base() + 3 * cap)[i]; }
    __device__ __forceinline__ uint16_t& PAR(uint32_t i) const {
        return reinterpret_cast<uint16_t*>(base() + 3 * cap)[2 * cap + i];
    }
};
struct GlobalRows {
    const MixBatch& b;
    uint32_t node0;
    __device__ __forceinline__ double& D(uint32_t i) const { return b.elimD[node0 + i]; }
    __device__ __forceinline__ double& R(uint32_t i) const { return b.elimR[node0 + i]; }
    __device__ __forceinline__ double* side(bool r) const { return (r ? b.elimR : b.elimD) + node0; }
    __device__ __forceinline__ double OFF(uint32_t i) const { return __ldg(b.off + node0 + i); }
    __device__ __forceinline__ uint32_t TOPO(uint32_t i) const { return __ldg(b.topo + node0 + i); }
    __device__ __forceinline__ uint32_t PAR(uint32_t i) const { return __ldg(b.par + node0 + i); }
};

struct HalfRows {                // D and R in shared memory (`cap` nodes), the rest global
    const MixBatch& b;
    uint32_t node0, slot, cap;
    __device__ __forceinline__ double& D(uint32_t i) const { return sArea()[slot + i]; }
    __device__ __forceinline__ double& R(uint32_t i) const { return sArea()[cap + slot + i]; }
    __device__ __forceinline__ double OFF(uint32_t i) const { return __ldg(b.off + node0 + i); }
    __device__ __forceinline__ uint32_t TOPO(uint32_t i) const { return __ldg(b.topo + node0 + i); }
    __device__ __forceinline__ uint32_t PAR(uint32_t i) const { return __ldg(b.par + node0 + i); }
};
// Forward elimination of node i: pull the children's eliminated rows (diag -=
// off_c * f_c, rhs -= off_c * g_c), then keep g = rhs/pivot in R and f =
// off/pivot in D.
template <class Rows>
__device__ __forceinline__ void pullNode(const Rows& E, uint32_t i) {
    const uint32_t t = E.TOPO(i);
    const uint32_t c0 = t & 0xFFFF, c1 = c0 + ((t >> 16) & 0xFF);
    double d = E.D(i), r = E.R(i);
    for (uint32_t c = c0; c < c1; ++c) {
        const double oc = E.OFF(c);
        d = fma(-oc, E.D(c), d);
        r = fma(-oc, E.R(c), r);
    }
    const double iv = rcpPivot(d);
    E.R(i) = r * iv;
    E.D(i) = E.OFF(i) * iv;
}

// A narrow level (at most half as many nodes, b0 .. e, as threads): two lanes
// per node, the even one on the pivot (D), the odd one on the right-hand
// side (R), so that each child costs one FP64 warp instruction instead of two
// (the FP64 cost is per warp instruction).
template <class Rows>
__device__ __forceinline__ void pullNarrow(const Rows& E, uint32_t b0, uint32_t e, uint32_t tid) {
    const uint32_t i = b0 + (tid >> 1);
    const bool rl = tid & 1u;
    const bool on = i < e;
    const uint32_t t = on ? E.TOPO(i) : 0u;
    const uint32_t c0 = t & 0xFFFF, c1 = c0 + ((t >> 16) & 0xFF);
    double* const a = E.side(rl);
    double x = on ? a[i] : 1.0;
    for (uint32_t c = c0; c < c1; ++c) x = fma(-E.OFF(c), a[c], x);
    const double ivd = rcpPivot(x);
    const double iv = __shfl_sync(0xFFFFFFFFu, ivd, (tid & 31u) & ~1u);
    const double y = (rl ? x : (on ? E.OFF(i) : 0.0)) * iv;
    if (on) a[i] = y;
}

// Per-cell work of tick 0 (stimulus schedule) for the forest's cells.
__device__ __forceinline__ void forestStimulus(const MixBatch& b, uint32_t cell0, uint32_t nCells,
                                               unsigned long long step, uint32_t t0, uint32_t nt) {
    for (uint32_t k = t0; k < nCells; k += nt) {
        const uint32_t cell = b.forestCells[cell0 + k];
        const MixCellRange cr = b.cells[cell];
        if (!cr.nStim || step >= stopOf(b, cell)) continue;
        uint32_t cur = b.stimCur[cell];
        while (cur < cr.nStim && b.stimStep[cr.stim0 + cur] <= step) {
            b.injVal[cr.inj0 + b.stimEntry[cr.stim0 + cur]] = b.stimValue[cr.stim0 + cur];
            ++cur;
        }
        b.stimCur[cell] = cur;
    }
}

// SpikeGens (SpikeGen::process with the solver's V and currTime = dt (step+1))
// and trace samples, one thread per cell.
__device__ __forceinline__ void forestOutputs(const MixBatch& b, uint32_t cell0, uint32_t nCells,
                                              unsigned long long step, uint32_t t0, uint32_t nt) {
    const double currTime = b.dt * (double)(step + 1);
    const bool sample = ((step + 1) % b.recStride) == 0;
    for (uint32_t k = t0; k < nCells; k += nt) {
        const uint32_t cell = b.forestCells[cell0 + k];
        if (step >= stopOf(b, cell)) continue;
        const MixCellRange cr = b.cells[cell];
        for (uint32_t g = cr.sg0; g < cr.sg0 + cr.nSg; ++g) {
            const double Vs = b.V[b.sgNode[g]];
            if (Vs > (double)b.sgThresh[g]) {
                if ((float)(currTime + b.dt / 2.0) >= b.sgLast[g] + b.sgRefract[g] && !(b.sgEdge[g] && b.sgFired[g])) {
                    const uint32_t spk = b.spikeCount[cell];
                    if (spk < b.spikeCap) {
                        b.spikeGen[(size_t)cell * b.spikeCap + spk] = g - cr.sg0;
                        b.spikeTime[(size_t)cell * b.spikeCap + spk] = (float)currTime;
                    }
                    b.spikeCount[cell] = spk + 1;
                    b.sgLast[g] = (float)currTime;
                    b.sgFired[g] = 1;
                }
            } else {
                b.sgFired[g] = 0;
            }
        }
        if (cr.nRec && sample) {
            const uint64_t smp = (step + 1) / b.recStride;
            if (smp < b.recCap)
                for (uint32_t r = cr.rec0; r < cr.rec0 + cr.nRec; ++r)
                    b.recBuf[smp * b.recLd + r] = b.V[b.recNode[r]];
        }
    }
}

// Bulk prefetch into L2 (cp.async.bulk.prefetch) of forest nodes
// [first, first + count) of per-node array `k`, clamped to the array and
// aligned to 16 bytes; called by one thread per array.
__device__ __forceinline__ void prefetchNodes(const MixBatch& b, uint32_t k, uint64_t first, uint32_t count) {
    const PrefetchArr a = b.pf[k];
    const uint64_t total = (uint64_t)a.n * a.elem / 16 * 16;
    uint64_t lo = first * a.elem / 16 * 16;
    uint64_t hi = ((first + count) * a.elem + 15) / 16 * 16;
    if (hi > total) hi = total;
    if (lo >= hi) return;
    const char* p = static_cast<const char*>(a.base) + lo;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"((uint32_t)(hi - lo)) : "memory");
}

// V = 2 VMid - V, then the node's Ca pool: the end of a step of one node.
__device__ __forceinline__ void updateNode(const MixBatch& b, uint32_t n, uint32_t info, double vm) {
    const double Vnew = fma(2.0, vm, -b.V[n]);
    b.V[n] = Vnew;
    if (info & kNodePool) {
        const float vca = (float)(b.caAdvance == 1 ? vm : fma(2.0, vm, -Vnew));
        const float act = fmaf(-b.caG[n], vca, b.caGE[n]);
        const float c0v = b.poolC[n];
        float c = fmaf(-b.poolG1[n], c0v, c0v) + b.poolF2[n] * act;
        float cav = b.poolBasal[n] + c;
        if (b.poolCeil[n] > 0.f && cav > b.poolCeil[n]) { cav = b.poolCeil[n]; c = cav - b.poolBasal[n]; }
        if (cav < b.poolFloor[n]) { cav = b.poolFloor[n]; c = cav - b.poolBasal[n]; }
        b.poolC[n] = c;
        b.poolCa[n] = cav;
    }
}

// After a forest's last step (`step` = steps done): that step's update and
// outputs, the per-cell step counts and the forest's counter.
template <class Rows>
__device__ __forceinline__ void finishForest(const MixBatch& b, uint32_t f, const Rows& E, unsigned long long step) {
    const MixForest F = b.forests[f];
    const uint32_t tid = threadIdx.x, nth = blockDim.x;
    for (uint32_t i = tid; i < F.nNodes; i += nth) {
        const uint32_t n = F.node0 + i;
        const uint32_t info = __ldg(b.nodeInfo + n);
        if (info & kNodeCenter) continue;
        if (step - 1 < stopOf(b, __ldg(b.cellOf + n))) updateNode(b, n, info, E.R(i));
    }
    __syncthreads();
    forestOutputs(b, F.cell0, F.nCells, step - 1, tid, nth);
    for (uint32_t k = tid; k < F.nCells; k += nth) {
        const uint32_t cell = b.forestCells[F.cell0 + k];
        const unsigned long long stop = stopOf(b, cell);
        b.stepCount[cell] = step < stop ? step : stop;
    }
    if (tid == 0) b.forestStep[f] = step;
    __syncthreads();
}

// `nsteps` steps of one forest by the whole CTA.  The V/Ca update and the
// outputs (SpikeGens, trace samples) of a step run at the start of the next
// step's assembly, and after the last step.  A cell whose stop step is
// reached stays as it is: its nodes get a neutral row (pivot 1, rhs 0) so
// that the elimination of the forest goes on around them.
template <bool kAhead, class Rows>
__device__ __forceinline__ void stepForest(const MixBatch& b, const MixForest& F, uint32_t f,
                                           const Rows& E, const uint32_t* lp, uint32_t nsteps) {
    const uint32_t tid = threadIdx.x, nth = blockDim.x;
    if (nsteps == 0) return;
    unsigned long long step = b.forestStep[f];
    // SynChans of the forest: [k0, k1).  Those of step 0 of the launch are
    // advanced here; those of every later step by the threads that a level of
    // the previous step's elimination leaves idle (whole idle warps take the
    // next synapses in order), the rest after that elimination.
    const uint32_t k0 = __ldg(b.syn0 + F.node0), k1 = __ldg(b.syn0 + F.node0 + F.nNodes);
    for (uint32_t k = k0 + tid; k < k1; k += nth) synapseStep(b, k, step);
    for (uint32_t s = 0; s < nsteps; ++s, ++step) {
        if (tid < b.nPf) prefetchNodes(b, tid, F.node0, nth);
        forestStimulus(b, F.cell0, F.nCells, step, tid, nth);
        __syncthreads();
        // assembly: every node's FP64 row (junction nodes: their diagonal);
        // the next chunk of nth nodes is prefetched into L2 meanwhile
        for (uint32_t i = tid; i < F.nNodes; i += nth) {
            if (tid < b.nPf && i + nth - tid < F.nNodes) prefetchNodes(b, tid, F.node0 + i + nth - tid, nth);
            const uint32_t n = F.node0 + i;
            const uint32_t info = __ldg(b.nodeInfo + n);
            const unsigned long long stop = b.anyStop ? b.stopStep[__ldg(b.cellOf + n)] : ~0ull;
            const bool live = step < stop;                  // this step advances the cell
            const bool pending = s > 0 && step - 1 < stop;  // the previous step's update
            double d = 1.0, r = 0.0;
            if (info & kNodeCenter) {
                if (live) d = __ldg(b.HS2 + n);
            } else if (live) {
                assembleNode<kAhead>(b, n, info, pending, pending ? E.R(i) : 0.0, d, r);
            } else if (pending) {
                updateNode(b, n, info, E.R(i));
            }
            E.D(i) = d;
            E.R(i) = r;
        }
        __syncthreads();
        if (s > 0) forestOutputs(b, F.cell0, F.nCells, step - 1, tid, nth);
        // forward elimination, deepest level first
        const bool ahead = s + 1 < nsteps;     // advance the next step's synapses
        uint32_t kNext = k0;
        for (int L = (int)F.nLevels - 1; L >= 0; --L) {
            const uint32_t b0 = lp[L], e = lp[L + 1];
            if (ahead && kNext < k1) {
                const uint32_t busy = (e - b0 + 31) & ~31u;
                if (busy < nth) {
                    if (tid >= busy && kNext + (tid - busy) < k1) synapseStep(b, kNext + (tid - busy), step + 1);
                    kNext += nth - busy;
                }
            }
            for (uint32_t i = b0 + tid; i < e; i += nth) pullNode(E, i);
            __syncthreads();
        }
        // back substitution, root level first: VMid = g - f * VMid[parent]
        for (uint32_t L = 0; L < F.nLevels; ++L) {
            const uint32_t e = lp[L + 1];
            for (uint32_t i = lp[L] + tid; i < e; i += nth) {
                const uint32_t p = E.PAR(i);
                double vm = E.R(i);
                if (p != kNoParent) vm = fma(-E.D(i), E.R(p), vm);
                E.R(i) = vm;
            }
            __syncthreads();
        }
        if (ahead)
            for (uint32_t k = kNext + tid; k < k1; k += nth) synapseStep(b, k, step + 1);
    }
    finishForest(b, f, E, step);
}

// Named barrier over `count` threads (a multiple of 32).
__device__ __forceinline__ void groupSync(uint32_t id, uint32_t count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// A counter in shared memory that orders what its threads wrote before
// (release) and read after (acquire), within the CTA: a full fence would also
// wait for the reads a thread has under way (in the eliminators of a cluster it
// took 6 to 18 us of a step: 9,001 compartments on 4 CTAs 122 us with, 103 without;
// 3,500 62 and 56).  kCluster: threads of the cluster's other CTAs add to it
// too, after a fence of cluster scope.
template <bool kCluster>
__device__ __forceinline__ uint32_t loadAcquire(const uint32_t* p) {
    uint32_t v;
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    if (kCluster) asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    else asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void addRelease(uint32_t* p, uint32_t v) {
    asm volatile("red.release.cta.shared::cta.add.u32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}

// Bounded wait of an eliminator for a level's assembly: at most
// b.waitRounds rounds of ~128 ns (default 2^24, far longer than any
// assembly), so that a lost update ends the kernel with an error instead of
// a hang.  A thread that gave up once, or that sees the batch's error flag
// set by another CTA, waits no more in this launch: the launch then ends
// after at most one bounded wait per eliminator thread, and its results are
// marked invalid (hs_batch_sync returns HS_ETIMEOUT).
template <bool kCluster = false>
__device__ __forceinline__ bool waitLevel(const MixBatch& b, const uint32_t* done, uint32_t need, bool& gaveUp) {
    if (gaveUp) return false;
    uint32_t rounds = 0;
    while (loadAcquire<kCluster>(done) < need) {
        ++rounds;
        if (rounds > b.waitRounds || ((rounds & 1023u) == 0 && *(volatile const uint32_t*)b.err)) {
            atomicExch(b.err, 1u);
            gaveUp = true;
            return false;
        }
        __nanosleep(128);
    }
    return true;
}

// The same steps as stepForest with the CTA split into two groups.  The
// first `elimWarps` warps eliminate; the others assemble nodes deepest level
// first and count the finished nodes of each level in `done` (shared
// memory).  The eliminators start a level of the forward elimination as soon
// as its count is complete, so the elimination of the deep levels overlaps
// the assembly of the shallow ones; meanwhile the assemblers emit the
// previous step's outputs and advance the next step's SynChans.  Then the
// whole CTA substitutes back.  Forests of fewer than kWsLevels levels.
template <bool kStops, bool kAhead, class Rows>
__device__ __forceinline__ void stepForestWS(const MixBatch& b, uint32_t f, const Rows& E, uint32_t elimWarps,
                                             uint32_t nsteps) {
    volatile const MixForest& F = sCtl().F;
    const uint32_t* lp = sLevels();
    uint32_t* done = sDone();
    const uint32_t tid = threadIdx.x, nth = blockDim.x;
    if (nsteps == 0) return;
    const uint32_t nE = 32 * elimWarps, nA = nth - nE;
    const bool elim = tid < nE;
    const uint32_t atid = tid - nE;
    if (tid == 0) {
        sCtl().step = b.forestStep[f];
        sCtl().syn0 = __ldg(b.syn0 + F.node0);
        sCtl().syn1 = __ldg(b.syn0 + F.node0 + F.nNodes);
    }
    __syncthreads();
    {
        const unsigned long long step = sCtl().step;
        for (uint32_t k = sCtl().syn0 + tid, k1 = sCtl().syn1; k < k1; k += nth) synapseStep(b, k, step);
    }
    bool gaveUp = false;
    for (uint32_t s = 0; s < nsteps; ++s) {
        for (uint32_t L = tid; L < F.nLevels; L += nth) done[L] = 0;
        forestStimulus(b, F.cell0, F.nCells, sCtl().step, tid, nth);
        __syncthreads();
        if (elim) {
            // forward elimination, each level once the assemblers finished it
            for (int L = (int)F.nLevels - 1; L >= 0; --L) {
                const uint32_t b0 = lp[L], e = lp[L + 1];
                waitLevel(b, &done[L], e - b0, gaveUp);
                if (2 * (e - b0) <= nE) {
                    pullNarrow(E, b0, e, tid);
                } else {
                    for (uint32_t i = b0 + tid; i < e; i += nE) pullNode(E, i);
                }
                groupSync(1, nE);
            }
        } else {
            // assembly, deepest level first (the highest node indices); each
            // node's info word is loaded one node ahead, which takes the
            // first of the node's dependent memory round trips off its chain
            const uint32_t node0 = F.node0;
            int i = (int)F.nNodes - 1 - (int)atid;
            uint32_t infoNext = i >= 0 ? __ldg(b.nodeInfo + node0 + i) : 0u;
            for (; i >= 0; i -= (int)nA) {
                if (atid < b.nPf && i + (int)atid >= (int)nA) {
                    const uint32_t hi = (uint32_t)i + atid + 1 - nA;     // next chunk: [hi - nA, hi)
                    prefetchNodes(b, atid, node0 + (hi > nA ? hi - nA : 0), hi > nA ? nA : hi);
                }
                const uint32_t n = node0 + i;
                const uint32_t info = infoNext;
                if (i >= (int)nA) infoNext = __ldg(b.nodeInfo + n - nA);
                bool live = true, pending = s > 0;
                if (kStops) {
                    const unsigned long long stop = stopOf(b, __ldg(b.cellOf + n)), step = sCtl().step;
                    live = step < stop;
                    pending = pending && step - 1 < stop;
                }
                double d = 1.0, r = 0.0;
                if (info & kNodeCenter) {
                    if (live) d = __ldg(b.HS2 + n);
                } else if (live) {
                    assembleNode<kAhead>(b, n, info, pending, pending ? E.R(i) : 0.0, d, r);
                } else if (pending) {
                    updateNode(b, n, info, E.R(i));
                }
                E.D(i) = d;
                E.R(i) = r;
                addRelease(&done[E.TOPO(i) >> 24], 1u);
            }
            groupSync(2, nA);
            const unsigned long long step = sCtl().step;
            if (s > 0) forestOutputs(b, F.cell0, F.nCells, step - 1, atid, nA);
            if (s + 1 < nsteps)
                for (uint32_t k = sCtl().syn0 + atid, k1 = sCtl().syn1; k < k1; k += nA) synapseStep(b, k, step + 1);
        }
        __syncthreads();
        if (tid == 0) sCtl().step = sCtl().step + 1;      // (read next after the barriers of the back substitution)
        // back substitution by the whole CTA
        const uint32_t nL = F.nLevels;
        if (F.shared == kRowsShared) {
            for (uint32_t L = 0; L < nL; ++L) {
                const uint32_t e = lp[L + 1];
                for (uint32_t i = lp[L] + tid; i < e; i += nth) {
                    const uint32_t p = E.PAR(i);
                    double vm = E.R(i);
                    if (p != kNoParent) vm = fma(-E.D(i), E.R(p), vm);
                    E.R(i) = vm;
                }
                __syncthreads();
            }
        } else {
            // in global memory: a thread's first node of the next level has
            // its parent index, coupling and right-hand side (none of which
            // this level changes) loaded before the barrier, leaving one
            // dependent load (the parent's value) per level
            uint32_t nb = lp[0] + tid, ne = lp[1], pn = 0;
            double dn = 0.0, rn = 0.0;
            if (nb < ne) {
                pn = E.PAR(nb);
                dn = E.D(nb);
                rn = E.R(nb);
            }
            for (uint32_t L = 0; L < nL; ++L) {
                const uint32_t i0 = nb, e = ne, p0 = pn;
                const double d0 = dn, r0 = rn;
                if (L + 1 < nL) {
                    nb = lp[L + 1] + tid;
                    ne = lp[L + 2];
                    if (nb < ne) {
                        pn = E.PAR(nb);
                        dn = E.D(nb);
                        rn = E.R(nb);
                    }
                }
                if (i0 < e) E.R(i0) = p0 != kNoParent ? fma(-d0, E.R(p0), r0) : r0;
                for (uint32_t i = i0 + nth; i < e; i += nth) {
                    const uint32_t p = E.PAR(i);
                    double vm = E.R(i);
                    if (p != kNoParent) vm = fma(-E.D(i), E.R(p), vm);
                    E.R(i) = vm;
                }
                __syncthreads();
            }
        }
    }
    finishForest(b, f, E, sCtl().step);
}

// The prototypes into shared memory; a barrier follows before they are read.
__device__ __forceinline__ void copyTypes(const MixBatch& b) {
    auto copy = [](const void* dst, const void* src, uint32_t bytes) {
        for (uint32_t i = threadIdx.x; i < bytes / 4; i += blockDim.x)
            static_cast<uint32_t*>(const_cast<void*>(dst))[i] = static_cast<const uint32_t*>(src)[i];
    };
    copy(sChanTypes(), b.chanTypes, kMaxChanTypes * sizeof(ChanType));
    copy(sC2dTypes(), b.c2dTypes, kMaxC2dTypes * sizeof(C2dType));
    copy(sSynTypes(), b.synTypes, kMaxSynTypes * sizeof(SynType));
}

// What the elimination of a node reads of its forest's constants in global
// memory: its topology word, its off-diagonal and its first two children's.
struct PullIn {
    uint32_t topo;
    double off;
    double2 offC;
};
__device__ __forceinline__ PullIn pullIn(const MixBatch& b, uint32_t n) {
    PullIn q;
    q.topo = __ldg(b.topo + n);
    q.off = __ldg(b.off + n);
    q.offC = __ldg(b.offC + n);
    return q;
}
// pullNode and pullNarrow of a half-shared forest, those constants at hand.
__device__ __forceinline__ void pullNode(const HalfRows& E, uint32_t i, const PullIn& q) {
    const uint32_t c0 = q.topo & 0xFFFF, nc = (q.topo >> 16) & 0xFF;
    double d = E.D(i), r = E.R(i);
    if (nc) {
        d = fma(-q.offC.x, E.D(c0), d);
        r = fma(-q.offC.x, E.R(c0), r);
        if (nc > 1) {
            d = fma(-q.offC.y, E.D(c0 + 1), d);
            r = fma(-q.offC.y, E.R(c0 + 1), r);
            for (uint32_t c = c0 + 2; c < c0 + nc; ++c) {
                const double oc = E.OFF(c);
                d = fma(-oc, E.D(c), d);
                r = fma(-oc, E.R(c), r);
            }
        }
    }
    const double iv = rcpPivot(d);
    E.R(i) = r * iv;
    E.D(i) = q.off * iv;
}
__device__ __forceinline__ void pullNarrow(const HalfRows& E, uint32_t i, bool on, uint32_t tid, const PullIn& q) {
    const bool rl = tid & 1u;
    double x = 1.0;
    if (on) {
        const uint32_t c0 = q.topo & 0xFFFF, nc = (q.topo >> 16) & 0xFF;
        const double* a = &E.D(0) + (rl ? E.cap : 0);
        x = a[i];
        if (nc) {
            x = fma(-q.offC.x, a[c0], x);
            if (nc > 1) {
                x = fma(-q.offC.y, a[c0 + 1], x);
                for (uint32_t c = c0 + 2; c < c0 + nc; ++c) x = fma(-E.OFF(c), a[c], x);
            }
        }
    }
    const double ivd = rcpPivot(x);
    const double iv = __shfl_sync(0xFFFFFFFFu, ivd, (tid & 31u) & ~1u);
    const double y = (rl ? x : q.off) * iv;
    if (on) (rl ? E.R(i) : E.D(i)) = y;
}

// This CTA's writes (global and shared) made visible at cluster scope.
__device__ __forceinline__ void fenceCluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }

// Forward elimination of a half-shared forest by threads t of nE (barrier
// `bar`), deepest level first, each once its rows are assembled.  What a node
// reads from global memory is read a node ahead, across the levels (a
// population of 1,024 cells 120 us per step, 140 without): on the chain are
// only the counter, the rows in shared memory and the arithmetic.
template <bool kCluster>
__device__ __forceinline__ void forwardHalf(const MixBatch& b, const HalfRows& E, uint32_t nL, const uint32_t* lp,
                                            const uint32_t* done, uint32_t t, uint32_t nE, uint32_t bar,
                                            bool& gaveUp) {
    uint32_t b0 = lp[nL - 1], e = lp[nL];
    uint32_t i = b0 + (2 * (e - b0) <= nE ? t >> 1 : t);
    PullIn q = {0, 0.0, {0.0, 0.0}};
    if (i < e) q = pullIn(b, E.node0 + i);
    for (int L = (int)nL - 1; L >= 0; --L) {
        const bool narrow = 2 * (e - b0) <= nE;
        waitLevel<kCluster>(b, &done[L], e - b0, gaveUp);
        for (;; i += nE) {
            const bool last = i + nE >= e;       // of this level
            const uint32_t i0 = i;
            const bool on = i < e;
            const PullIn q0 = q;
            if (!last) {
                q = pullIn(b, E.node0 + i + nE);
            } else {
                if (L > 0) {
                    const uint32_t nb = lp[L - 1];
                    i = nb + (2 * (b0 - nb) <= nE ? t >> 1 : t);
                    if (i < b0) q = pullIn(b, E.node0 + i);
                    e = b0;
                    b0 = nb;
                }
            }
            if (narrow) pullNarrow(E, i0, on, t, q0);
            else if (on) pullNode(E, i0, q0);
            if (last) break;
        }
        groupSync(bar, nE);
    }
}

// Its back substitution, root level first, by threads t of nt; a node's parent
// index and row, none of which the level above changes, are read a node ahead.
__device__ __forceinline__ void backHalf(const HalfRows& E, uint32_t nL, const uint32_t* lp, uint32_t t, uint32_t nt,
                                         uint32_t bar) {
    uint32_t nb = lp[0] + t, ne = lp[1], pn = 0;
    double dn = 0.0, rn = 0.0;
    if (nb < ne) {
        pn = E.PAR(nb);
        dn = E.D(nb);
        rn = E.R(nb);
    }
    for (uint32_t L = 0; L < nL; ++L) {
        for (;;) {
            const uint32_t i0 = nb, e0 = ne, p0 = pn;
            const double d0 = dn, r0 = rn;
            const bool last = nb + nt >= ne;
            if (!last) nb += nt;
            else if (L + 1 < nL) {
                nb = lp[L + 1] + t;
                ne = lp[L + 2];
            }
            if (nb < ne) {
                pn = E.PAR(nb);
                dn = E.D(nb);
                rn = E.R(nb);
            }
            if (i0 < e0) E.R(i0) = p0 != kNoParent ? fma(-d0, E.R(p0), r0) : r0;
            if (last) break;
        }
        groupSync(bar, nt);
    }
}

// Offsets and counters of the levels of forest g of a pair (fewer than
// kWsLevels), in sLevels' words.
__device__ __forceinline__ uint32_t* pairLevels(uint32_t g) { return sLevels() + g * kWsLevels; }
__device__ __forceinline__ uint32_t* pairDone(uint32_t g) { return sLevels() + (2 + g) * kWsLevels; }
static_assert(4 * kWsLevels <= kSmemLevels, "room for a pair's levels");

// The steps of stepForestWS for two forests at once (or, groups == 1, one), half
// shared: each has its own group of `elimWarps` eliminators, all other warps
// assemble the one, then the other, deepest level first.  While a forest is
// eliminated, its outputs are emitted and it is substituted back by its
// eliminators, the assemblers are at the other.
// Bound by the assembly's memory latency and, in the eliminators' chains, by
// the FP64 pipe they share with it: a population of 1,024 cells (8,850 nodes a
// CTA) takes 112 us per step, 140 as two shared forests stepped one after the
// other, where the assemblers idle through the end of each elimination.
// Barrier 4 + g, before each assembly of forest g, is met by its eliminators
// (VMid of the last step is there, the counters are zero) and by all
// assemblers; so a forest's SynChans and stimulus, advanced before it, follow
// the other forest's barrier and with it the assembly that read the old ones
// (of a lone forest, barrier 3).
template <bool kStops>
__device__ __forceinline__ void stepPair(const MixBatch& b, uint32_t groups, uint32_t halfCap, uint32_t elimWarps,
                                         uint32_t nsteps) {
    const uint32_t tid = threadIdx.x, nth = blockDim.x;
    const uint32_t nE = 32 * elimWarps, nA = nth - groups * nE;
    if (tid < groups * nE) {
        const uint32_t g = tid >= nE ? 1 : 0, t = tid - g * nE;
        volatile ForestCtl& C = sCtl(g);
        const HalfRows E{b, C.F.node0, C.F.slot, halfCap};
        const uint32_t* lp = pairLevels(g);
        uint32_t* done = pairDone(g);
        bool gaveUp = false;
        for (uint32_t s = 0; s < nsteps; ++s) {
            __threadfence_block();
            groupSync(4 + g, nE + nA);
            const uint32_t nL = C.F.nLevels;
            forwardHalf<false>(b, E, nL, lp, done, t, nE, 1 + g, gaveUp);
            for (uint32_t L = t; L < nL; L += nE) done[L] = 0;
            if (s > 0) forestOutputs(b, C.F.cell0, C.F.nCells, C.step + s - 1, t, nE);
            backHalf(E, nL, lp, t, nE, 1 + g);
        }
    } else {
        const uint32_t atid = tid - groups * nE;
        for (uint32_t q = 0; q < groups * nsteps; ++q) {
            const uint32_t s = groups == 2 ? q >> 1 : q, g = groups == 2 ? q & 1 : 0;
            volatile ForestCtl& C = sCtl(g);
            if (groups == 1) groupSync(3, nA);
            if (atid < b.nPf) {
                const uint32_t n = C.F.nNodes, m = min(n, nA);
                prefetchNodes(b, atid, C.F.node0 + n - m, m);
            }
            forestStimulus(b, C.F.cell0, C.F.nCells, C.step + s, atid, nA);
            for (uint32_t k = C.syn0 + atid, k1 = C.syn1; k < k1; k += nA) synapseStep(b, k, C.step + s);
            groupSync(4 + g, nE + nA);
            const uint32_t node0 = C.F.node0;
            const HalfRows E{b, node0, C.F.slot, halfCap};
            uint32_t* done = pairDone(g);
            int i = (int)C.F.nNodes - 1 - (int)atid;
            uint32_t infoNext = i >= 0 ? __ldg(b.nodeInfo + node0 + i) : 0u;
            for (; i >= 0; i -= (int)nA) {
                if (atid < b.nPf && i + (int)atid >= (int)nA) {
                    const uint32_t hi = (uint32_t)i + atid + 1 - nA;     // next chunk: [hi - nA, hi)
                    prefetchNodes(b, atid, node0 + (hi > nA ? hi - nA : 0), hi > nA ? nA : hi);
                }
                const uint32_t n = node0 + i;
                const uint32_t info = infoNext;
                if (i >= (int)nA) infoNext = __ldg(b.nodeInfo + n - nA);
                bool live = true, pending = s > 0;
                if (kStops) {
                    const unsigned long long stop = stopOf(b, __ldg(b.cellOf + n)), step = C.step + s;
                    live = step < stop;
                    pending = pending && step - 1 < stop;
                }
                double d = 1.0, r = 0.0;
                if (info & kNodeCenter) {
                    if (live) d = __ldg(b.HS2 + n);
                } else if (live) {
                    assembleNode<true>(b, n, info, pending, pending ? E.R(i) : 0.0, d, r);
                } else if (pending) {
                    updateNode(b, n, info, E.R(i));
                }
                E.D(i) = d;
                E.R(i) = r;
                const uint32_t level = __ldg(b.topo + n) >> 24;
                const uint32_t act = __activemask(), first = __ffs(act) - 1, L0 = __shfl_sync(act, level, first);
                if (__all_sync(act, level == L0)) {
                    __syncwarp(act);
                    if ((tid & 31u) == first) addRelease(&done[level], __popc(act));
                } else {
                    addRelease(&done[level], 1u);
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t g = 0; g < groups; ++g) {
        volatile ForestCtl& C = sCtl(g);
        const HalfRows E{b, C.F.node0, C.F.slot, halfCap};
        finishForest(b, C.forest, E, C.step + nsteps);
    }
}

// One CTA steps its half-shared forests, in pairs where MixForest::mate says so
// (a lone forest has both groups' warps to eliminate); fewer than kWsLevels
// levels each.  D of forest node i is double slot + i after the level offsets,
// R lies `halfCap` doubles further.
template <bool kStops>
__global__ void __launch_bounds__(1024, 1) hsForestPairStepMixed(MixBatch b, const uint32_t* __restrict__ ctaPtr,
                                                                 const uint32_t* __restrict__ ctaForests,
                                                                 uint32_t halfCap, uint32_t elimWarps,
                                                                 uint32_t nsteps) {
    if (nsteps == 0) return;
    copyTypes(b);
    const uint32_t k1 = ctaPtr[blockIdx.x + 1];
    for (uint32_t k = ctaPtr[blockIdx.x], groups; k < k1; k += groups) {
        groups = 1 + b.forests[ctaForests[k]].mate;
        if (kStops) {      // (all cells stopped: as in hsForestStepMixed)
            bool over = true;
            for (uint32_t g = 0; g < groups; ++g)
                over = over && b.forestStep[ctaForests[k + g]] >= b.forestStop[ctaForests[k + g]];
            if (over) {
                __syncthreads();
                if (threadIdx.x < groups) b.forestStep[ctaForests[k + threadIdx.x]] += nsteps;
                continue;
            }
        }
        for (uint32_t g = 0; g < groups; ++g) {
            const uint32_t f = ctaForests[k + g], level0 = b.forests[f].level0, nL = b.forests[f].nLevels;
            for (uint32_t i = threadIdx.x; i <= nL; i += blockDim.x) {
                pairLevels(g)[i] = b.levelPtr[level0 + i];
                pairDone(g)[i] = 0;
            }
            if (threadIdx.x == 0) {
                const MixForest F = b.forests[f];
                volatile ForestCtl& C = sCtl(g);
                C.F.node0 = F.node0;
                C.F.nNodes = F.nNodes;
                C.F.nLevels = F.nLevels;
                C.F.cell0 = F.cell0;
                C.F.nCells = F.nCells;
                C.F.slot = F.slot + kDeepDoubles;
                C.forest = f;
                C.step = b.forestStep[f];
                C.syn0 = __ldg(b.syn0 + F.node0);
                C.syn1 = __ldg(b.syn0 + F.node0 + F.nNodes);
            }
        }
        __syncthreads();
        stepPair<kStops>(b, groups, halfCap, groups == 1 ? 2 * elimWarps : elimWarps, nsteps);
    }
}

// OFF, TOPO and PAR of forest F into shared memory; a barrier follows before
// they are read.
__device__ __forceinline__ void stageForest(const MixBatch& b, const MixForest& F, const SharedRows& E) {
    for (uint32_t i = threadIdx.x; i < F.nNodes; i += blockDim.x) {
        E.OFF(i) = b.off[F.node0 + i];
        E.TOPO(i) = b.topo[F.node0 + i];
        E.PAR(i) = b.par[F.node0 + i];
    }
}

// One CTA steps its forests one after the other, each for `nsteps` steps.
// Dynamic shared memory: the header, then for shared forests the elimination
// arrays of `cap` nodes: D, R, OFF (8 B each), TOPO (4 B), PAR (2 B); for
// half-shared ones D and R of `cap` nodes.  `deep`: doubles before them that
// belong to the level offsets.
// `elimWarps`, `globalWarps`: eliminators of a forest in shared and in global
// memory.
// kStops: the batch has stop steps (b.anyStop); kSteps: how its forests are
// stepped, kSplit (stepForestWS), kUnsplit (stepForest: 256 levels or more, or
// no eliminator warps), or some each way; kModes: where their arrays may be
// (bits 1 << kRows*).  Registers are what a thread has least of: 1,024 threads
// get 64 each, and a spill costs an L2 access, the L1 being what shared memory
// leaves (304 cables of 300 compartments 207 us per step, 251 with the split
// step in the same kernel), so a batch gets the instantiation with no more in
// it than its forests need.
constexpr uint32_t kSplit = 1, kUnsplit = 2;      // bits of kSteps
template <bool kStops, uint32_t kSteps, uint32_t kModes>
__global__ void __launch_bounds__(1024, 1) hsForestStepMixed(MixBatch b, const uint32_t* __restrict__ ctaPtr,
                                                             const uint32_t* __restrict__ ctaForests, uint32_t cap,
                                                             uint32_t deep, uint32_t elimWarps,
                                                             uint32_t globalWarps, uint32_t nsteps) {
    constexpr bool kAhead = kSteps != (kSplit | kUnsplit) && (kModes & (kModes - 1)) == 0;
    copyTypes(b);
    for (uint32_t k = ctaPtr[blockIdx.x]; k < ctaPtr[blockIdx.x + 1]; ++k) {
        const MixForest F = b.forests[ctaForests[k]];
        if (kStops && b.forestStep[ctaForests[k]] >= b.forestStop[ctaForests[k]]) {
            // every cell of the forest has reached its stop step: stepping it
            // would change nothing (stopped cells keep their state, outputs
            // and step counts), so its steps are only counted and the CTA
            // can return and free its SM for other batches
            __syncthreads();
            if (threadIdx.x == 0) b.forestStep[ctaForests[k]] += nsteps;
            continue;
        }
        const uint32_t* lp = b.levelPtr + F.level0;
        if (F.nLevels < kWsLevels + 2 * deep) {
            for (uint32_t i = threadIdx.x; i <= F.nLevels; i += blockDim.x) sLevels()[i] = lp[i];
            lp = sLevels();
        }
        const SharedRows S{cap, deep};
        const GlobalRows G{b, F.node0};
        if (F.shared == kRowsShared) stageForest(b, F, S);
        if (threadIdx.x == 0) {
            volatile MixForest& c = sCtl().F;
            c.node0 = F.node0;
            c.nNodes = F.nNodes;
            c.nLevels = F.nLevels;
            c.cell0 = F.cell0;
            c.nCells = F.nCells;
            c.shared = F.shared;
        }
        __syncthreads();
        const uint32_t f = ctaForests[k];
        auto plain = [&](uint32_t warps) {
            return kSteps == kUnsplit ||
                   (kSteps != kSplit && !(warps && F.nLevels < kWsLevels && blockDim.x > 32 * warps));
        };
        if ((kModes & 1u << kRowsShared) && F.shared == kRowsShared) {
            if (plain(elimWarps)) stepForest<kAhead>(b, F, f, S, lp, nsteps);
            else stepForestWS<kStops, kAhead>(b, f, S, elimWarps, nsteps);
        } else if (kModes & 1u << kRowsHalf) {
            stepForest<kAhead>(b, F, f, HalfRows{b, F.node0, F.slot + deep, cap}, lp, nsteps);
        } else if (kModes & 1u << kRowsGlobal) {
            if (plain(globalWarps)) stepForest<kAhead>(b, F, f, G, lp, nsteps);
            else stepForestWS<kStops, kAhead>(b, f, G, globalWarps, nsteps);
        }
    }
}

// Reinit, per node: V = initVm, gates at their steady state, Ca = CaBasal,
// synapses, K(Ca) X.
__global__ void hsReinitNodesMixed(MixBatch b, uint32_t nNodes, const double* __restrict__ initVm,
                                   const float* __restrict__ k2x0, const uint32_t* __restrict__ evStart) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nNodes) return;
    const uint64_t ld = b.ld;
    const uint32_t info = b.nodeInfo[n];
    b.V[n] = initVm[n];
    if (info & kNodeCenter) return;
    if (info & kNodePool) {
        b.poolC[n] = 0.f;
        b.poolCa[n] = b.poolBasal[n];
    }
    const float ca = (info & kNodePool) ? b.poolCa[n] : 0.f;
    RowF vr = rowF(b.vTab, b.vCol, b.vRows, (float)initVm[n], b.vMin, b.vMax, b.vInvDx);
    const uint32_t types = b.ctype4[n];
    for (int j = 0; j < kMaxChan; ++j) {
        const uint32_t tj = (types >> (8 * j)) & 0xFF;
        if (tj == kNoType) break;
        const ChanType t = chanType(b, tj);
        float2* st = b.state + (uint64_t)(3 * j) * ld + n;
        const float2 z0 = make_float2(0.f, 0.f);
        if (t.xp) st[0] = gateStep(lookupF(vr, t.colX), z0, 0.f, 0.f, true);
        if (t.yp) st[ld] = gateStep(lookupF(vr, t.colY), z0, 0.f, 0.f, true);
        if (t.zp) {
            if (t.zCa)
                st[2 * ld] = gateStep(lookupF(rowF(b.caTab, b.caCol, b.caRows, ca, b.caMin, b.caMax, b.caInvDx),
                                              t.colZ), z0, 0.f, 0.f, true);
            else
                st[2 * ld] = gateStep(lookupF(vr, t.colZ), z0, 0.f, 0.f, true);
        }
    }
    if (((info >> 8) & kNoK2) != kNoK2) b.k2x[n] = k2x0[n];
    if (info & kNodeSyn)
        for (uint32_t k = b.syn0[n]; k < b.syn0[n + 1]; ++k) {
            b.synX[k] = 0.f;
            b.synY[k] = 0.f;
            b.evCur[k] = evStart[k];
        }
}

// Reinit, per cell: SpikeGens, counters, trace sample 0 (after the nodes).
__global__ void hsReinitCellsMixed(MixBatch b) {
    const uint32_t cell = blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= b.nCells) return;
    const MixCellRange cr = b.cells[cell];
    for (uint32_t g = cr.sg0; g < cr.sg0 + cr.nSg; ++g) {
        b.sgLast[g] = -b.sgRefract[g];
        b.sgFired[g] = 0;
    }
    if (cell < b.nForests) b.forestStep[cell] = 0;
    b.stepCount[cell] = 0;
    b.stimCur[cell] = 0;
    b.spikeCount[cell] = 0;
    for (uint32_t r = cr.rec0; r < cr.rec0 + cr.nRec; ++r) b.recBuf[r] = b.V[b.recNode[r]];
}

// Scatter of host-supplied inject values to their solver slots.
__global__ void hsScatterInject(double* const* __restrict__ addr, uint8_t* const* __restrict__ flag,
                                const double* __restrict__ val, uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    *addr[i] = val[i];
    if (flag[i]) *flag[i] = 1;
}

__global__ void hsScatterValues(const ValueWrite* __restrict__ w, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const ValueWrite x = w[i];
    if (x.f32) *static_cast<float*>(x.addr) = (float)x.value;
    else *static_cast<double*>(x.addr) = x.value;
}

cudaError_t launchScatterValues(const ValueWrite* w, uint32_t n, cudaStream_t st) {
    if (!n) return cudaSuccess;
    hsScatterValues<<<(n + 255) / 256, 256, 0, st>>>(w, n);
    return cudaGetLastError();
}

cudaError_t launchScatterInject(double* const* addr, uint8_t* const* flag, const double* val, uint32_t n,
                                cudaStream_t st) {
    if (!n) return cudaSuccess;
    hsScatterInject<<<(n + 255) / 256, 256, 0, st>>>(addr, flag, val, n);
    return cudaGetLastError();
}

// ---- several SMs per forest: a thread-block cluster -------------------------------
// For latency: the forests of one cluster of kC CTAs are stepped by all of
// them together.  A forest's pivots/couplings D and right-hand sides R live
// in rank 0's shared memory (16 B a node; of a large forest the rest stays in global
// memory); every CTA assembles (rank 0's first `elimWarps` warps excepted),
// writing each node's row into rank 0's D and R through distributed shared
// memory and adding the per-level completion counts there.  Rank 0's
// eliminator warps walk the levels as in stepForestWS, then rank 0 alone
// substitutes back.  The CTAs of the cluster meet at bounded barriers
// (clusterMeet) twice per step: after assembly and elimination, and after the
// back substitution (by when rank 0 has also reset the level counters and
// applied the next step's stimulus).  The arithmetic of every node is
// that of the one-CTA step, so results are bit-identical.

// A bounded barrier of the kC CTAs of a cluster on a counter in rank 0's
// shared memory (`bar`, a distributed shared memory address): each CTA adds
// 1 and waits for the count of this meeting, `gen` x kC.  Every wait is
// bounded by b.waitRounds sleeps; after a timeout, or once the batch's error
// flag is set, a CTA waits no more in this launch (the launch then ends with
// its results marked invalid, as with waitLevel).
__device__ __forceinline__ void clusterMeet(const MixBatch& b, uint32_t* bar, uint32_t& gen, uint32_t kC,
                                            bool& gaveUp) {
    __syncthreads();
    ++gen;
    if (threadIdx.x == 0) {
        fenceCluster();
        atomicAdd(bar, 1u);
        uint32_t rounds = 0;
        while (!gaveUp && *(volatile const uint32_t*)bar < gen * kC) {
            ++rounds;
            if (rounds > b.waitRounds || ((rounds & 1023u) == 0 && *(volatile const uint32_t*)b.err)) {
                atomicExch(b.err, 1u);
                gaveUp = true;
                break;
            }
            __nanosleep(64);
        }
        fenceCluster();
    }
    __syncthreads();
}

// `nsteps` steps of forest F by the cluster.  dR0 and rR0: D and R in rank
// 0's shared memory; E: the rows there, as rank 0 eliminates them.
template <bool kStaged, bool kAhead, class Rows>
__device__ __forceinline__ void stepForestCluster(const MixBatch& b, const MixForest& F, uint32_t f,
                                  const Rows& E, double* dR0, double* rR0, uint32_t* doneR0, uint32_t* barR0,
                                  uint32_t& gen, uint32_t rank, uint32_t kC, uint32_t elimWarps, uint32_t nsteps,
                                  bool& gaveUp) {
    const uint32_t* lp = sLevels();
    uint32_t* done = sDone();
    const uint32_t tid = threadIdx.x, nth = blockDim.x;
    const uint32_t nE = rank == 0 ? 32 * elimWarps : 0;
    const bool elim = tid < nE;
    const uint32_t nAL = nth - 32 * elimWarps;              // assemblers of rank 0
    const uint32_t ga = rank == 0 ? tid - nE : nAL + (rank - 1) * nth + tid;
    const uint32_t T = nAL + (kC - 1) * nth;                // assemblers of the cluster
    const uint32_t gt = rank * nth + tid, GT = kC * nth;     // every thread of the cluster
    unsigned long long step = b.forestStep[f];
    const uint32_t k0 = __ldg(b.syn0 + F.node0), k1 = __ldg(b.syn0 + F.node0 + F.nNodes);
    for (uint32_t k = k0 + gt; k < k1; k += GT) synapseStep(b, k, step);
    bool waitGaveUp = false;
    // each step's level counters and stimulus are set before the meeting
    // that ends the step before it (here, for the first step)
    if (rank == 0) {
        for (uint32_t L = tid; L < F.nLevels; L += nth) done[L] = 0;
        forestStimulus(b, F.cell0, F.nCells, step, tid, nth);
    }
    clusterMeet(b, barR0, gen, kC, gaveUp);
    for (uint32_t s = 0; s < nsteps; ++s, ++step) {
        if (elim) {
            if constexpr (!kStaged) {
                forwardHalf<true>(b, E, F.nLevels, lp, done, tid, nE, 1, waitGaveUp);
            } else {
                for (int L = (int)F.nLevels - 1; L >= 0; --L) {
                    const uint32_t b0 = lp[L], e = lp[L + 1];
                    waitLevel<true>(b, &done[L], e - b0, waitGaveUp);
                    if (2 * (e - b0) <= nE) {
                        pullNarrow(E, b0, e, tid);
                    } else {
                        for (uint32_t i = b0 + tid; i < e; i += nE) pullNode(E, i);
                    }
                    groupSync(1, nE);
                }
            }
        } else {
            for (uint32_t j = ga; j < F.nNodes; j += T) {
                const uint32_t i = F.nNodes - 1 - j;
                if (ga < b.nPf && j + T - ga < F.nNodes) {
                    const uint32_t hi = F.nNodes - (j + T - ga);
                    prefetchNodes(b, ga, F.node0 + (hi > T ? hi - T : 0), hi > T ? T : hi);
                }
                const uint32_t n = F.node0 + i;
                const uint32_t info = __ldg(b.nodeInfo + n);
                const unsigned long long stop = b.anyStop ? b.stopStep[__ldg(b.cellOf + n)] : ~0ull;
                const bool live = step < stop;
                const bool pending = s > 0 && step - 1 < stop;
                double d = 1.0, r = 0.0;
                if (info & kNodeCenter) {
                    if (live) d = __ldg(b.HS2 + n);
                } else if (live) {
                    assembleNode<kAhead>(b, n, info, pending, pending ? rR0[i] : 0.0, d, r);
                } else if (pending) {
                    updateNode(b, n, info, rR0[i]);
                }
                dR0[i] = d;
                rR0[i] = r;
                fenceCluster();
                atomicAdd(doneR0 + (__ldg(b.topo + n) >> 24), 1u);
            }
        }
        clusterMeet(b, barR0, gen, kC, gaveUp);
        // the previous step's outputs (the update ran in this assembly), the
        // next step's SynChans, then rank 0 substitutes back
        if (rank == 0 && s > 0) forestOutputs(b, F.cell0, F.nCells, step - 1, tid, nth);
        if (s + 1 < nsteps)
            for (uint32_t k = k0 + gt; k < k1; k += GT) synapseStep(b, k, step + 1);
        if (rank == 0) {
            __syncthreads();
            if constexpr (!kStaged) {
                backHalf(E, F.nLevels, lp, tid, nth, 0);
            } else {
                for (uint32_t L = 0; L < F.nLevels; ++L) {
                    const uint32_t e = lp[L + 1];
                    for (uint32_t i = lp[L] + tid; i < e; i += nth) {
                        const uint32_t p = E.PAR(i);
                        double vm = E.R(i);
                        if (p != kNoParent) vm = fma(-E.D(i), E.R(p), vm);
                        E.R(i) = vm;
                    }
                    __syncthreads();
                }
            }
            if (s + 1 < nsteps) {
                for (uint32_t L = tid; L < F.nLevels; L += nth) done[L] = 0;
                forestStimulus(b, F.cell0, F.nCells, step + 1, tid, nth);
            }
        }
        clusterMeet(b, barR0, gen, kC, gaveUp);
    }
    if (rank == 0) finishForest(b, f, E, step);
    clusterMeet(b, barR0, gen, kC, gaveUp);
}

// Forests of cluster blockIdx.x / kC (ctaPtr/ctaForests per cluster), each
// of at most `cap` nodes and kWsLevels - 1 levels (the host packs them so).
// Dynamic shared memory: the header, then the forest's D and R (used in rank
// 0): a forest of at most `stageCap` nodes also gets OFF, TOPO and PAR there
// (30 B a node, like a one-CTA shared forest), a larger one keeps them in
// global memory (D and R only, 16 B a node, up to `cap` nodes).
// kModes: staged forests (kRowsShared), larger ones (kRowsHalf), as above.
template <uint32_t kModes>
__global__ void __launch_bounds__(1024, 1) hsForestStepMixedCluster(MixBatch b, const uint32_t* __restrict__ ctaPtr,
                                                                    const uint32_t* __restrict__ ctaForests,
                                                                    uint32_t kC, uint32_t cap, uint32_t stageCap,
                                                                    uint32_t elimWarps, uint32_t nsteps) {
    constexpr bool kAhead = (kModes & (kModes - 1)) == 0;
    copyTypes(b);
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    if (threadIdx.x == 0) *sBarrier() = 0;
    for (uint32_t L = threadIdx.x; L < kWsLevels; L += blockDim.x) sDone()[L] = 0;
    cluster.sync();                                   // rank 0's counters are set before anyone adds
    uint32_t* doneR0 = cluster.map_shared_rank(sDone(), 0);
    uint32_t* barR0 = cluster.map_shared_rank(sBarrier(), 0);
    uint32_t gen = 0;
    bool gaveUp = false;
    const uint32_t c = blockIdx.x / kC;
    for (uint32_t k = ctaPtr[c]; k < ctaPtr[c + 1]; ++k) {
        const uint32_t f = ctaForests[k];
        const MixForest F = b.forests[f];
        for (uint32_t i = threadIdx.x; i <= F.nLevels; i += blockDim.x) sLevels()[i] = b.levelPtr[F.level0 + i];
        const bool stage = F.nNodes <= stageCap;
        const SharedRows S{stageCap, 0};
        const HalfRows H{b, F.node0, 0, cap};
        if (stage && rank == 0) stageForest(b, F, S);
        __syncthreads();
        double* const d = cluster.map_shared_rank(sArea(), 0);
        if ((kModes & 1u << kRowsShared) && stage)
            stepForestCluster<true, kAhead>(b, F, f, S, d, d + stageCap, doneR0, barR0, gen, rank, kC, elimWarps, nsteps, gaveUp);
        else if (kModes & 1u << kRowsHalf)
            stepForestCluster<false, kAhead>(b, F, f, H, d, d + cap, doneR0, barR0, gen, rank, kC, elimWarps, nsteps, gaveUp);
    }
    cluster.sync();                                   // rank 0's shared memory outlives every remote access
}

// One launch of the cluster kernel: nClusters clusters of kC CTAs.
cudaError_t launchForestStepMixedCluster(const MixBatch& b, const uint32_t* ctaPtr, const uint32_t* ctaForests,
                                         uint32_t nClusters, uint32_t kC, uint32_t threadsPerCta,
                                         uint32_t smemBytes, uint32_t cap, uint32_t stageCap, uint32_t elimWarps,
                                         uint32_t modes, uint32_t nsteps, cudaStream_t st) {
    constexpr uint32_t S = 1u << kRowsShared, H = 1u << kRowsHalf;
    auto kern = modes == S ? hsForestStepMixedCluster<S>
                           : modes == H ? hsForestStepMixedCluster<H> : hsForestStepMixedCluster<S | H>;
    cudaError_t e = allowShared((const void*)kern);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nClusters * kC);
    cfg.blockDim = dim3(threadsPerCta);
    cfg.dynamicSmemBytes = smemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kC;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, b, ctaPtr, ctaForests, kC, cap, stageCap, elimWarps,
                              nsteps);
}

cudaError_t launchForestStepMixed(const MixBatch& b, const uint32_t* ctaPtr, const uint32_t* ctaForests,
                                  uint32_t nCtas, uint32_t threadsPerCta, uint32_t smemBytes, uint32_t cap,
                                  uint32_t deep, uint32_t pairWarps, uint32_t elimWarps, uint32_t globalWarps,
                                  uint32_t minLevels, uint32_t maxLevels, uint32_t modes, uint32_t nsteps,
                                  cudaStream_t st) {
    // maxLevels: the deepest forest's levels; modes: bits 1 << MixForest::shared
    if (pairWarps) {
        auto kern = b.anyStop ? hsForestPairStepMixed<true> : hsForestPairStepMixed<false>;
        cudaError_t e = allowShared((const void*)kern);
        if (e != cudaSuccess) return e;
        kern<<<nCtas, threadsPerCta, smemBytes, st>>>(b, ctaPtr, ctaForests, cap, pairWarps, nsteps);
        return cudaGetLastError();
    }
    const uint32_t warps = std::max(elimWarps, globalWarps);
    constexpr uint32_t S = 1u << kRowsShared, G = 1u << kRowsGlobal;
    auto kern = b.anyStop ? hsForestStepMixed<true, kSplit | kUnsplit, S | G>
                          : hsForestStepMixed<false, kSplit | kUnsplit, S | G>;
    if (elimWarps && maxLevels < kWsLevels && threadsPerCta > 32 * warps) {
        if (modes == S) kern = b.anyStop ? hsForestStepMixed<true, kSplit, S> : hsForestStepMixed<false, kSplit, S>;
        else if (modes == G) kern = b.anyStop ? hsForestStepMixed<true, kSplit, G> : hsForestStepMixed<false, kSplit, G>;
        else kern = b.anyStop ? hsForestStepMixed<true, kSplit, S | G> : hsForestStepMixed<false, kSplit, S | G>;
    } else if (!elimWarps || minLevels >= kWsLevels || threadsPerCta <= 32 * std::min(elimWarps, globalWarps)) {
        kern = modes == S ? hsForestStepMixed<true, kUnsplit, S> : hsForestStepMixed<true, kUnsplit, S | G>;
    }
    if (modes == 1u << kRowsHalf) kern = hsForestStepMixed<true, kUnsplit, 1u << kRowsHalf>;
    cudaError_t e = allowShared((const void*)kern);
    if (e != cudaSuccess) return e;
    kern<<<nCtas, threadsPerCta, smemBytes, st>>>(b, ctaPtr, ctaForests, cap, deep, elimWarps, globalWarps, nsteps);
    return cudaGetLastError();
}

cudaError_t launchBatchReinitMixed(const MixBatch& b, uint32_t nNodes, const double* initVm, const float* k2x0,
                                   const uint32_t* evStart, cudaStream_t st) {
    hsReinitNodesMixed<<<(nNodes + 255) / 256, 256, 0, st>>>(b, nNodes, initVm, k2x0, evStart);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const uint32_t n = b.nCells > b.nForests ? b.nCells : b.nForests;
    hsReinitCellsMixed<<<(n + 127) / 128, 128, 0, st>>>(b);
    return cudaGetLastError();
}

}  // namespace hsg
