// hs_fp64.cu -- the FP64 drop-in HSolve step on GB300 (sm_103a).
//
// One CTA steps one cell for `nsteps` clock steps without returning to the
// host.  Per step, in the reference's tick order (scheduling/Clock.cpp:872-921):
//   tick 0   basal-inject schedule
//   tick 1/4 SimpleSynHandler -> SynChan, HHChannel2D  (one thread per object)
//   tick 6   HSolveActive::step (hsolve/HSolveActive.cpp:45-66):
//            advanceChannels + calculateChannelCurrents + updateMatrix
//            (one thread per compartment), forward elimination and back
//            substitution (level by level over the pull programs, the rows
//            of a level shared by the CTA; cable runs by one thread),
//            advanceCalcium (one thread per pool), SpikeGens, trace record.
// Compiled with --fmad=false: every operation is the reference's IEEE
// operation in the reference's order, so Vm/Ca are bit-identical to the CPU
// HSolve wherever no libm call is involved (exp/log only in HHChannel2D and
// non-integer gate powers).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/moose_gb300.h"
#include "hs_device.cuh"
#include "hs_plan.h"
#include "hs_shared.h"

namespace hsg {

// ---- tick 1: external calcium (DifShell, DifBuffer, MMPump) ----------------
// biophysics/DifShell.cpp, biophysics/DifBuffer.cpp, biophysics/MMPump.cpp.
// The objects process in tick order and each send reaches its targets at
// once (a target later in the same tick sees this step's value), so one
// thread walks them in order.  State: kDifState arrays of nDif (see DevCell).
namespace dif {
constexpr double kF = 96485.3415;                 // DifShell::F
constexpr double kEpsilon = 1.0e-10;              // DifShell/DifBuffer::EPSILON
constexpr double kPi = 3.14159265358979323846;    // M_PI
enum { C_ = 0, PREVC, DC, CM, BFREE, BBOUND, PREVFREE, AF, BF, ACT, VOL, OUTERA, INNERA };
}  // namespace dif

__device__ __forceinline__ double& difS(const DevCell& c, int field, uint32_t k) {
    return c.difState[(size_t)field * c.nDif + k];
}
__device__ __forceinline__ double difP(const DevCell& c, uint32_t k, int i) {
    return c.difPar[(size_t)k * HS_DIF_NPAR + i];
}

// DifShell::calculateVolumeArea, DifBuffer::vReinit's geometry
__device__ void difGeometry(const DevCell& c, uint32_t k) {
    using namespace dif;
    const int shape = (int)difP(c, k, 4);
    const double length = difP(c, k, 5), diameter = difP(c, k, 6), thickness = difP(c, k, 7);
    const double rOut = diameter / 2.;
    double rIn = rOut - thickness;
    if (rIn < 0) rIn = 0.;
    if (shape == 0) {
        if (length == 0.0) {
            difS(c, VOL, k) = 4. / 3. * kPi * (rOut * rOut * rOut - rIn * rIn * rIn);
            difS(c, OUTERA, k) = 4 * kPi * rOut * rOut;
            difS(c, INNERA, k) = 4 * kPi * rIn * rIn;
        } else {
            difS(c, VOL, k) = (kPi * length) * (rOut * rOut - rIn * rIn);
            difS(c, OUTERA, k) = 2 * kPi * rOut * length;
            difS(c, INNERA, k) = 2 * kPi * rIn * length;
        }
    } else if (shape == 1) {
        difS(c, VOL, k) = kPi * diameter * diameter * thickness / 4.0;
        difS(c, OUTERA, k) = kPi * diameter * diameter / 4.0;
        difS(c, INNERA, k) = difS(c, OUTERA, k);
    } else {
        difS(c, VOL, k) = difP(c, k, 8);
        difS(c, OUTERA, k) = difP(c, k, 9);
        difS(c, INNERA, k) = difP(c, k, 10);
    }
}

__device__ __forceinline__ double difIntegrate(double state, double dt, double A, double B) {
    if (B > dif::kEpsilon) {
        const double x = exp(-B * dt);
        return state * x + (A / B) * (1 - x);
    }
    return state + A * dt;
}

// inner/outerDifSourceOut of object s: fluxFromIn/Out of each target
__device__ void difSendFlux(const DevCell& c, uint32_t s, int kind, double value, double thickness) {
    using namespace dif;
    const uint32_t slot = s * kDifMsgKinds + kind;
    for (uint32_t i = c.difOff[slot]; i < c.difOff[slot + 1]; ++i) {
        const uint32_t t = c.difDst[i];
        const bool shell = c.difKind[t] == HS_DIF_SHELL;
        const double D = shell ? difP(c, t, 1) : difP(c, t, 3);
        const double area = kind == HS_DMSG_OUTER ? difS(c, OUTERA, t) : difS(c, INNERA, t);
        const double tt = difP(c, t, 7);
        if (shell) {
            const double diff = 2. * D / difS(c, VOL, t) * area / (thickness + tt);
            difS(c, DC, t) += diff * value;
            difS(c, CM, t) += diff;
        } else {
            const double d = 2 * D / difS(c, VOL, t) * area / (tt + thickness);
            difS(c, AF, t) += d * value;
            difS(c, BF, t) += d;
        }
    }
}

// concentrationOut of shell s: HHChannel concen (HSolve::addConc) and DifBuffer
// concentration (its activation)
__device__ void difSendConc(const DevCell& c, uint32_t s, double C) {
    uint32_t slot = s * kDifMsgKinds + HS_DMSG_CONC_CHAN;
    for (uint32_t i = c.difOff[slot]; i < c.difOff[slot + 1]; ++i) c.extCa[c.difDst[i]] = C;
    slot = s * kDifMsgKinds + HS_DMSG_CONC_BUF;
    for (uint32_t i = c.difOff[slot]; i < c.difOff[slot + 1]; ++i) difS(c, dif::ACT, c.difDst[i]) = C;
}

// DifShell::vReinit, DifBuffer::vReinit (MMPump::reinit does nothing)
__device__ void difReinit(const DevCell& c) {
    using namespace dif;
    for (uint32_t k = 0; k < c.nDif; ++k) {
        const int kind = c.difKind[k];
        if (kind == HS_DIF_SHELL) {
            difS(c, DC, k) = difP(c, k, 3);
            difS(c, CM, k) = 0;
            difGeometry(c, k);
            difS(c, C_, k) = difP(c, k, 0);
            difS(c, PREVC, k) = difP(c, k, 0);
            difSendConc(c, k, difS(c, C_, k));
            difSendFlux(c, k, HS_DMSG_INNER, difS(c, PREVC, k), difP(c, k, 7));
            difSendFlux(c, k, HS_DMSG_OUTER, difS(c, PREVC, k), difP(c, k, 7));
        } else if (kind == HS_DIF_BUFFER) {
            difS(c, AF, k) = 0;
            difS(c, BF, k) = 0;
            difGeometry(c, k);
            const double bTot = difP(c, k, 0), kf = difP(c, k, 1), kb = difP(c, k, 2);
            difS(c, BFREE, k) = bTot / (1 + difS(c, ACT, k) * kf / kb);
            difS(c, PREVFREE, k) = difS(c, BFREE, k);
            difS(c, BBOUND, k) = bTot - difS(c, BFREE, k);
            difSendFlux(c, k, HS_DMSG_INNER, difS(c, PREVFREE, k), difP(c, k, 7));
            difSendFlux(c, k, HS_DMSG_OUTER, difS(c, PREVFREE, k), difP(c, k, 7));
        }
    }
}

// DifShell::vProcess, DifBuffer::vProcess, MMPump::process
__device__ void difProcess(const DevCell& c) {
    using namespace dif;
    for (uint32_t k = 0; k < c.nDif; ++k) {
        const int kind = c.difKind[k];
        if (kind == HS_DIF_SHELL) {
            difS(c, C_, k) = difIntegrate(difS(c, C_, k), c.dt, difS(c, DC, k), difS(c, CM, k));
            difS(c, DC, k) = difP(c, k, 3);
            difS(c, CM, k) = 0;
            difS(c, PREVC, k) = difS(c, C_, k);
            difSendFlux(c, k, HS_DMSG_INNER, difS(c, PREVC, k), difP(c, k, 7));
            difSendFlux(c, k, HS_DMSG_OUTER, difS(c, PREVC, k), difP(c, k, 7));
            difSendConc(c, k, difS(c, C_, k));
        } else if (kind == HS_DIF_BUFFER) {
            const double bTot = difP(c, k, 0), kf = difP(c, k, 1), kb = difP(c, k, 2);
            difS(c, AF, k) += kb * difS(c, BBOUND, k);
            difS(c, BF, k) += kf * difS(c, ACT, k);
            difS(c, BFREE, k) = difIntegrate(difS(c, BFREE, k), c.dt, difS(c, AF, k), difS(c, BF, k));
            difS(c, BBOUND, k) = bTot - difS(c, BFREE, k);
            difS(c, PREVFREE, k) = difS(c, BFREE, k);
            difSendFlux(c, k, HS_DMSG_INNER, difS(c, PREVFREE, k), difP(c, k, 7));
            difSendFlux(c, k, HS_DMSG_OUTER, difS(c, PREVFREE, k), difP(c, k, 7));
            const uint32_t slot = k * kDifMsgKinds + HS_DMSG_REACTION;     // reactionOut -> DifShell::vBuffer
            for (uint32_t i = c.difOff[slot]; i < c.difOff[slot + 1]; ++i) {
                const uint32_t t = c.difDst[i];
                difS(c, DC, t) += kb * difS(c, BBOUND, k);
                difS(c, CM, t) += kf * difS(c, BFREE, k);
            }
            difS(c, AF, k) = 0;
            difS(c, BF, k) = 0;
        } else {
            const double vMax = difP(c, k, 0), Kd = difP(c, k, 1);
            const uint32_t slot = k * kDifMsgKinds + HS_DMSG_PUMP;          // PumpOut -> DifShell::vMMPump
            for (uint32_t i = c.difOff[slot]; i < c.difOff[slot + 1]; ++i) {
                const uint32_t t = c.difDst[i];
                difS(c, CM, t) += (vMax / difS(c, VOL, t)) / (difS(c, C_, t) + Kd);
            }
        }
    }
}

// HSolveActive::sendValues, IkOut (hsolve/HSolveActive.cpp:367-376):
// (Ek - Vm) Gk of each channel, channel order, to DifShell::vInflux
__device__ void difSendIk(const DevCell& c) {
    for (uint32_t q = 0; q < c.C; ++q) {
        if (c.ikOff[q] == c.ikOff[q + 1]) continue;
        const double I = (c.Ek[q] - c.V[c.chanCompt[q]]) * c.Gk[q];
        for (uint32_t i = c.ikOff[q]; i < c.ikOff[q + 1]; ++i) {
            const uint32_t t = c.ikDst[i];
            difS(c, dif::DC, t) += I / (dif::kF * difP(c, t, 2) * difS(c, dif::VOL, t));
        }
    }
}

// ---- tick 1/4: external objects -------------------------------------------
__device__ __forceinline__ void synchanStep(const DevCell& c, uint32_t k, double currTime) {
    // SimpleSynHandler::vProcess: deliver events with time <= currTime
    double activation = 0.0;
    uint32_t e = c.evCur[k], end = c.evPtr[k + 1];
    while (e < end && atMost(c.evTime[e], currTime)) {
        activation += c.evW[e] / c.dt;
        ++e;
    }
    c.evCur[k] = e;
    double act = c.synAct[k];
    if (!isZero(activation)) act += activation;
    // SynChan::calcGk
    double X = act * c.synXc1[k] + c.synX[k] * c.synXc2[k];
    double Y = X * c.synYc1[k] + c.synY[k] * c.synYc2[k];
    c.synX[k] = X;
    c.synY[k] = Y;
    c.synAct[k] = 0.0;
    c.synGk[k] = Y * c.synNorm[k] * c.synMod[k];
}

__device__ __forceinline__ double depValue(uint32_t dep, double vm, double c1, double c2) {
    return dep == 0 ? vm : dep == 1 ? c1 : dep == 2 ? c2 : 0.0;
}

// HHChannel2D k on the inputs vm, c1, c2; its Gk.
__device__ __forceinline__ double chan2dStep(const DevCell& c, uint32_t k, double vm, double c1, double c2) {
    double g = c.c2dGbar[k];
    const uint32_t a = c.c2dA[k];
    if (a & 15u) {
        const int gi = c.c2dGate[k];
        const double x = depValue((a >> 4) & 15u, vm, c1, c2);
        const double y = depValue((a >> 8) & 15u, vm, c1, c2);
        double A, B;
        interp2dBoth(c.g2dAB + c.g2dOff[gi], c.g2dGeom + 6 * gi, c.g2dN[2 * gi],
                     c.g2dN[2 * gi + 1], x, y, A, B);
        double X = c.c2dX[k];
        if ((a >> 12) & 1u) {
            X = plainQuotient(A, B);
        } else if (lessThan(1.0e-10, B)) {   // HHChannelBase::integrate (exponential Euler)
            const double e = exp(-B * c.dt);
            X = X * e + quotient(A, B) * (1 - e);
        } else {
            X = X + A * c.dt;
        }
        c.c2dX[k] = X;
        g *= takePower(X, a & 15u, c.c2dXpow + k);
    }
    const double mod = c.c2dMod[k];
    if (!isOne(mod)) {
        keepBranch();
        g *= mod;
    }
    c.c2dGk[k] = g;
    return g;
}

// ---- tick 6, per compartment: channels + matrix row -----------------------
// Bound by the FP64 pipe (76 cycles per warp instruction and sub-partition):
// the gates run in one loop over X, Y, Z, and what is not an operation of the
// reference's arithmetic (compares, row indices, powers of 1, factors of 1)
// is kept off that pipe.  `first`: the launch's first step, the only one
// with conductances and currents sent between process calls and with
// HHChannel2D inputs that may differ from V and Ca (a field written since
// they were sent).  `own2d`: the HHChannel2Ds of the compartment are stepped
// here.  The row goes to M (diagonal at ic, right-hand side at N + ic).
__device__ __forceinline__ void rowStep(const DevCell& c, uint32_t ic, double hdt, bool own2d, bool first, bool last,
                                        double* M) {
    const double V = c.V[ic];
    const Row vRow = tableRow(V, c.vMin, c.vMax, c.vDx, c.vRdx, c.vRows);
    double GkSum = 0.0, GkEkSum = 0.0;
    for (uint32_t q = c.chanPtr[ic]; q < c.chanPtr[ic + 1]; ++q) {
        const uint4 A = c.chanA[q];
        const int inst = c.instant[q];
        double fraction = c.mod[q];
        bool one = isOne(fraction);
        uint32_t s = A.y;
        int32_t col = (int32_t)A.z;
        for (uint32_t g = 0; g < 3; ++g) {      // X, Y, Z (ChannelStruct::process multiplies in that order)
            const uint32_t code = (A.x >> (4 * g)) & 15u;
            if (code) {
                Row r = vRow;
                const double* T = c.vTab;
                uint32_t nCol = c.vCol;
                if (g == 2) {
                    const int32_t src = c.zSrc[q];
                    col = c.colZ[q];
                    const double ca = src >= 0 ? c.ca[src] : c.extCa[q];
                    if (src >= 0 || lessThan(0.0, ca)) {
                        r = tableRow(ca, c.caMin, c.caMax, c.caDx, c.caRdx, c.caRows);
                        T = c.caTab;
                        nCol = c.caCol;
                    }
                }
                double C1, C2;
                tableLookup(T, nCol, col, r, C1, C2);
                const double x = gateStep(c.state[s], C1, C2, c.dt, hdt, inst & (1 << g));
                c.state[s++] = x;
                double pw = takePower(x, code, (g == 0 ? c.Xpow : g == 1 ? c.Ypow : c.Zpow) + q);
                if (!one) {
                    keepBranch();
                    pw = fraction * pw;
                }
                fraction = pw;
                one = false;
            }
            col = (int32_t)A.w;
        }
        const double gk = c.Gbar[q] * fraction;
        c.Gk[q] = gk;
        GkSum += gk;
        GkEkSum += gk * c.Ek[q];
    }
    // external conductances in tick-4 send order (HSolve::addGkEk)
    double eg = 0.0, ege = 0.0, inj = 0.0;
    if (first) {
        eg = c.ext[2 * ic];
        ege = c.ext[2 * ic + 1];
        inj = c.injVarying[ic];
        c.ext[2 * ic] = 0.0;
        c.ext[2 * ic + 1] = 0.0;
        c.injVarying[ic] = 0.0;
    }
    for (uint32_t k = c.extPtr[ic]; k < c.extPtr[ic + 1]; ++k) {
        const int32_t code = c.extList[k];
        double gk, ek;
        if (code >= 0) {
            ek = c.c2dEk[code];
            if (!own2d) {
                gk = c.c2dGk[code];
            } else {
                const int32_t p1 = c.c2dConc1[code], p2 = c.c2dConc2[code];
                const bool sent = first;
                gk = chan2dStep(c, code, sent ? c.c2dVm[code] : V, sent || p1 < 0 ? c.c2dC1[code] : c.ca[p1],
                                sent || p2 < 0 ? c.c2dC2[code] : c.ca[p2]);
            }
        } else {
            gk = c.synGk[-code - 1];
            ek = c.synEk[-code - 1];
        }
        eg += gk;
        ege += gk * ek;
    }
    if (last) {
        c.prevExt[2 * ic] = eg;
        c.prevExt[2 * ic + 1] = ege;
    }
    // HSolveActive::updateMatrix
    double diag = c.HS2[ic] + GkSum;
    double rhs = V * c.CmByDt[ic] + c.EmByRm[ic] + GkEkSum;
    if (c.injPresent[ic]) {
        keepBranch();
        rhs += inj + c.injBasal[ic];
    }
    diag += eg;
    rhs += ege;
    M[ic] = diag;
    M[c.N + ic] = rhs;
}

// ---- advanceCalcium, per pool ----------------------------------------------
// V already holds the step's new value.  `first`: a current sent by `iCa`
// since the last process call may be waiting.
__device__ __forceinline__ void poolStep(const DevCell& c, uint32_t p, const double* VMid, bool first) {
    double act = 0.0;
    if (first) {
        act = c.iCa[p];
        c.iCa[p] = 0.0;
    }
    for (uint32_t f = c.feedPtr[p]; f < c.feedPtr[p + 1]; ++f) {
        uint32_t q = c.feedChan[f];
        uint32_t ic = c.chanCompt[q];
        const double v = c.caAdvance == 1 ? VMid[ic] : __fma_rn(2.0, VMid[ic], -c.V[ic]);
        act += c.Gk[q] * (c.Ek[q] - v);
    }
    double cc = c.f1[p] * c.c[p] + c.f2[p] * act;
    double ca = c.CaBasal[p] + cc;
    if (lessThan(0.0, c.ceil[p]) && lessThan(c.ceil[p], ca)) {
        ca = c.ceil[p];
        cc = ca - c.CaBasal[p];
    }
    if (lessThan(ca, c.floor_[p])) {
        ca = c.floor_[p];
        cc = ca - c.CaBasal[p];
    }
    c.c[p] = cc;
    c.ca[p] = ca;
}

// The end of a step of compartment ic: V = 2 VMid - V (2 VMid is exact) and
// its pools.
__device__ __forceinline__ void finishCompt(const DevCell& c, uint32_t ic, const double* VMid, bool first) {
    c.V[ic] = __fma_rn(2.0, VMid[ic], -c.V[ic]);
    for (uint32_t p = c.poolPtr[ic]; p < c.poolPtr[ic + 1]; ++p) poolStep(c, p, VMid, first);
}

// ---- elimination -------------------------------------------------------------
// Threads that step a cell together: a CTA, or a part of one with its own
// named barrier.
struct Team {
    uint32_t tid, nth, bar;
};
__device__ __forceinline__ void teamSync(const Team& t) {
    asm volatile("bar.sync %0, %1;" ::"r"(t.bar), "r"(t.nth) : "memory");
}

// A run of cable rows (one row per level, see CellPlan::fRun/bRun) is walked
// by one lane with the pivot's values carried in registers, the row
// indices computed (row r: diagonal M[r], right-hand side M[N + r],
// off-diagonal to r + 1 at off[r]) and the next row's operands loaded
// ahead; the operations and their order are those of the general loop.
__device__ __forceinline__ void forwardCableRun(double* M, const double* off, uint32_t N, uint32_t r, uint32_t run) {
    double d = M[r - 1], rhs = M[N + r - 1];
    double o1 = off[r - 1], dNext = M[r], rNext = M[N + r];
    for (uint32_t i = 0; i < run; ++i, ++r) {
        const double o = o1, dr = dNext, rr = rNext;
        if (i + 1 < run) {
            o1 = off[r];
            dNext = M[r + 1];
            rNext = M[N + r + 1];
        }
        const double q = quotient(o, d);
        d = dr - q * o;
        rhs = rr - q * rhs;
        M[r] = d;
        M[N + r] = rhs;
    }
}

__device__ __forceinline__ void backwardCableRun(const double* M, const double* off, double* VMid, uint32_t N,
                                                 uint32_t i, uint32_t run) {
    double vNext = VMid[i + 1];
    double rhs = M[N + i], o1 = off[i], diag = M[i];
    for (uint32_t j = 0; j < run; ++j, --i) {
        const double r = rhs, o = o1, dg = diag;
        if (j + 1 < run) {
            rhs = M[N + i - 1];
            o1 = off[i - 1];
            diag = M[i - 1];
        }
        double v = r;
        v -= o * vNext;
        v = quotient(v, dg);
        VMid[i] = v;
        vNext = v;
    }
}

// A long run shared by the lanes of a warp, with the serial walk's results.
// Each lane walks a piece of the run from a guess of the value that enters
// it, with the reference's operations; then every lane whose entry value is
// not, bit for bit, the one its left neighbour came out with walks again
// from that, until none is left.  By induction the first k pieces are final
// after k rounds (the first starts from the given value), so the result is
// the serial walk's whatever the guesses, in at most as many rounds as there
// are pieces.  It takes few because a cable's sweeps forget: an error in a
// pivot shrinks by q^2 per row, in a right-hand side or a voltage by q (the
// quotient, ~0.67 on the 201-compartment cable), and once it is below half a
// last place the two walks coincide.
// A lone lane's row is bound by latency (~670 cycles forward, ~490 back) and an
// FP64 instruction costs the same for one lane or 32: the 201-compartment
// cable's sweeps take 134k + 98k cycles per step row by row, 32k + 21k shared.
// From 64 rows: below that a piece is two rows or fewer.
constexpr uint32_t kWarmRows = 20;      // rows before a piece that its FP32 guess of the pivot walks

// Value of x as a float, cut; 0 outside the float range.
__device__ __forceinline__ float cutFloat(double x) {
    const uint32_t h = hiOf(x), e = (h >> 20) & 0x7FFu;
    const uint32_t b = ((h & 0x7FFFFFFFu) - 0x38000000u) << 3 | loOf(x) >> 29;
    return e - 897u < 253u ? __uint_as_float(b | (h & 0x80000000u)) : 0.f;
}

// Rounds of `walk(entry) -> exit` over the lanes' pieces; `active`: the lane
// has one.  Returns with every piece walked from its left neighbour's exit.
template <class Walk>
__device__ __forceinline__ void settle(double entry, bool active, Walk walk) {
    const uint32_t lane = threadIdx.x & 31u;
    double out = entry;
    bool go = active;
    for (uint32_t round = 0; round < 33; ++round) {
        if (go) out = walk(entry);
        const double left = __shfl_up_sync(0xFFFFFFFFu, out, 1);
        go = active && lane && bitsOf(left) != bitsOf(entry);
        if (go) entry = left;
        if (!__any_sync(0xFFFFFFFFu, go)) break;
    }
}

// Entry values of the pieces from their affine maps x -> a x + b, x0 entering
// the first (guesses, in plain FP64).
__device__ __forceinline__ double affineEntry(double a, double b, double x0) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k = 1; k < 32; k <<= 1) {
        const double pa = __shfl_up_sync(0xFFFFFFFFu, a, k), pb = __shfl_up_sync(0xFFFFFFFFu, b, k);
        if (lane >= k) {
            b = __fma_rn(a, pb, b);
            a = a * pa;
        }
    }
    const double end = __fma_rn(a, x0, b), left = __shfl_up_sync(0xFFFFFFFFu, end, 1);
    return lane ? left : x0;
}

// Rows r .. r + run - 1 forward; `S`: scratch of 2 run doubles.
__device__ __forceinline__ void forwardWarpRun(double* M, const double* off, uint32_t N, uint32_t r, uint32_t run,
                                               double* S) {
    const uint32_t lane = threadIdx.x & 31u, m = ((run + 31) / 32) | 1u;      // odd: no bank conflicts
    const uint32_t s = min(lane * m, run), e = min(s + m, run);
    const bool active = s < e;
    const double d0 = M[r - 1];
    double guess = d0;
    if (lane && active) {
        const uint32_t w = s > kWarmRows ? s - kWarmRows : 0u;
        float x = w ? cutFloat(M[r + w - 1]) : cutFloat(d0);
        for (uint32_t i = w; i < s; ++i) {
            const float o = cutFloat(off[r + i - 1]);
            x = cutFloat(M[r + i]) - __fdividef(o * o, x);
        }
        const uint32_t b = __float_as_uint(x);
        guess = fromWords((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + 0x38000000u), b << 29);
    }
    double* Q = S + run;
    settle(guess, active, [&](double d) {
        double oNext = off[r + s - 1], dNext = M[r + s];
        for (uint32_t i = s; i < e; ++i) {
            const double o = oNext, dr = dNext;
            if (i + 1 < e) {
                oNext = off[r + i];
                dNext = M[r + i + 1];
            }
            const double q = quotient(o, d);
            d = dr - q * o;
            S[i] = d;
            Q[i] = q;
        }
        return d;
    });
    for (uint32_t i = s; i < e; ++i) M[r + i] = S[i];
    // right-hand sides, with the quotients at hand
    double a = 1.0, b = 0.0;
    for (uint32_t i = s; i < e; ++i) {
        b = __fma_rn(-Q[i], b, M[N + r + i]);
        a = -Q[i] * a;
    }
    settle(affineEntry(a, b, M[N + r - 1]), active, [&](double x) {
        double qNext = Q[s], rNext = M[N + r + s];
        for (uint32_t i = s; i < e; ++i) {
            const double q = qNext, rr = rNext;
            if (i + 1 < e) {
                qNext = Q[i + 1];
                rNext = M[N + r + i + 1];
            }
            x = rr - q * x;
            S[i] = x;
        }
        return x;
    });
    for (uint32_t i = s; i < e; ++i) M[N + r + i] = S[i];
    __syncwarp();
}

// Rows i0, i0 - 1, .. (run of them) back; VMid over the right-hand sides.
__device__ __forceinline__ void backwardWarpRun(double* M, const double* off, uint32_t N, uint32_t i0, uint32_t run,
                                                double* S) {
    const uint32_t lane = threadIdx.x & 31u, m = ((run + 31) / 32) | 1u;
    const uint32_t s = min(lane * m, run), e = min(s + m, run);
    const bool active = s < e;
    double* R = M + N;
    double a = 1.0, b = 0.0;
    for (uint32_t j = s; j < e; ++j) {
        const double d = M[i0 - j];
        const Recip y = recip(d);
        const double q = quotient(off[i0 - j], d, y);
        b = __fma_rn(-q, b, quotient(R[i0 - j], d, y));
        a = -q * a;
    }
    settle(affineEntry(a, b, R[i0 + 1]), active, [&](double x) {
        double rNext = R[i0 - s], oNext = off[i0 - s], dNext = M[i0 - s];
        for (uint32_t j = s; j < e; ++j) {
            const double rr = rNext, o = oNext, d = dNext;
            if (j + 1 < e) {
                rNext = R[i0 - j - 1];
                oNext = off[i0 - j - 1];
                dNext = M[i0 - j - 1];
            }
            x = quotient(rr - o * x, d);
            S[j] = x;
        }
        return x;
    });
    for (uint32_t j = s; j < e; ++j) R[i0 - j] = S[j];
    __syncwarp();
}

// The level program of the forward sweep, for cells without waves (cables):
// a row's updates in order, the rows of a level shared by the team.
// `S`: scratch of the cell's runs in shared memory (DevCell::runRows), or null.
__device__ __forceinline__ void forwardLevels(const DevCell& c, double* M, const Team& t, double* S) {
    const uint32_t N = c.N, offBase = 2 * N + c.H;
    const double* off = c.M + offBase;
    auto at = [&](int32_t e) { return (uint32_t)e >= offBase ? off[e - offBase] : M[e]; };
    for (uint32_t l = 0; l < c.fLevels; ++l) {
        if (const uint32_t run = c.fRun[l]) {
            if (S && run >= kWarpRun) {
                if (t.tid < 32) forwardWarpRun(M, off, N, c.fRunRow[l], run, S);
            } else if (t.tid == 0) {
                forwardCableRun(M, off, N, c.fRunRow[l], run);
            }
            teamSync(t);
            l += run - 1;
            continue;
        }
        for (uint32_t k = c.fLevelPtr[l] + t.tid; k < c.fLevelPtr[l + 1]; k += t.nth) {
            // t -= l / pivot * a.  A row's consecutive updates by one pivot
            // (its diagonal and right-hand side: the reference computes
            // HS[4i+1] / HS[4i] for both) share the quotient: it is computed
            // once, the same IEEE division of the same operands.
            int32_t ql = -1, qp = -1;
            double q = 0.0;
            for (uint32_t o = c.fOpPtr[k]; o < c.fOpPtr[k + 1]; ++o) {
                int4 op = c.fOps[o];
                if (op.y != ql || op.w != qp) {
                    q = quotient(at(op.y), M[op.w]);
                    ql = op.y;
                    qp = op.w;
                }
                M[op.x] -= q * at(op.z);
                if (op.x == ql || op.x == qp) ql = -1;   // an operand changed
            }
        }
        teamSync(t);
    }
}

// Forward elimination and back substitution in shared memory: M holds the
// diagonal [0, N), the right-hand side [N, 2N), which becomes VMid, and the
// junction entries [2N, 2N + H); the off-diagonals, which never change, come
// with the updates' descriptors.
// A wave or level is one dependent chain: loads, a division, a product and a
// difference, a store, a barrier.  Two things follow.  A warp alone issues an
// instruction every ~4 cycles of it, so the narrow ones -- at most 16 updates
// or 32 rows, most of a cell's -- have a program of one record per lane, laid
// out wave after wave: no bounds, no loop, no branch but the division's rare
// one, and each of the two entries an update changes on a lane of its own
// (each with the quotient).  The first warp walks them without a barrier;
// the others call `idle` once meanwhile.  And a warp issues in order, so a
// load whose address waits for another load would hold up the chain: records
// are read one ahead from an address that is known.
// 500 branched compartments, one CTA, cycles per wave or level: ~2,300 in
// global memory, ~1,600 with per-wave bounds in shared memory.
constexpr uint32_t kNoIndex = 0xFFFFu;      // no second entry, no update or row for this lane
constexpr uint32_t kOffIndex = 0xFFFEu;     // the update's (row's) off-diagonal

struct ProgOp {
    uint4 d;        // the DevCell::fW or bW entry
    double off;     // its off-diagonal
    uint32_t t3;    // bW: the fourth term
};
__device__ __forceinline__ ProgOp progOp(const uint4* prog, uint32_t k) {
    ProgOp w;
    w.d = __ldg(prog + 2 * k);
    const uint4 o = __ldg(prog + 2 * k + 1);
    w.off = fromWords(o.y, o.x);
    w.t3 = o.z;
    return w;
}
__device__ __forceinline__ void waveEntry(double* M, uint32_t ta, double q, double off) {
    const uint32_t t = ta & 0xFFFFu, a = ta >> 16;
    if (t != kNoIndex) M[t] -= q * (a == kOffIndex ? off : M[a]);
}
__device__ __forceinline__ double waveQuotient(const double* M, const ProgOp& u) {
    const uint32_t l = u.d.z & 0xFFFFu;
    return quotient(l == kOffIndex ? u.off : M[l], M[u.d.z >> 16]);
}
// One entry of an update: {t | a << 16, l | p << 16, off-diagonal}.
__device__ __forceinline__ void laneUpdate(double* M, const uint4& r) {
    const uint32_t t = r.x & 0xFFFFu, a = r.x >> 16, l = r.y & 0xFFFFu;
    if (t == kNoIndex) return;
    const double off = fromWords(r.w, r.z), x = M[t];
    const double av = a == kOffIndex ? off : M[a], lv = l == kOffIndex ? off : M[l];
    M[t] = x - quotient(lv, M[r.y >> 16]) * av;
}
// A row: {row | terms << 16, the first three terms}, {off-diagonal, fourth
// term, first of the others in bX}.
__device__ __forceinline__ void substitute(const DevCell& c, double* M, const uint4* prog, uint32_t k, const ProgOp& b) {
    const uint32_t N = c.N, i = b.d.x & 0xFFFFu, n = b.d.x >> 16, co = b.d.y & 0xFFFFu;
    double v = M[N + i];
    const double d = M[i];
    if (n) {
        v -= (co == kOffIndex ? b.off : M[co]) * M[N + (b.d.y >> 16)];
        if (n > 1) v -= M[b.d.z & 0xFFFFu] * M[N + (b.d.z >> 16)];
        if (n > 2) v -= M[b.d.w & 0xFFFFu] * M[N + (b.d.w >> 16)];
        if (n > 3) v -= M[b.t3 & 0xFFFFu] * M[N + (b.t3 >> 16)];
        if (n > 4) {
            const uint32_t x0 = __ldg(prog + 2 * k + 1).w;
            for (uint32_t t = 4; t < n; ++t) {
                const uint32_t x = __ldg(c.bX + x0 + t - 4);
                v -= M[x & 0xFFFFu] * M[N + (x >> 16)];
            }
        }
    }
    M[N + i] = quotient(v, d);
}

template <class Idle>
__device__ __forceinline__ void eliminateShared(const DevCell& c, double* M, const Team& t, Idle idle) {
    const uint32_t N = c.N, lane = t.tid & 31u;
    const bool w0 = t.tid < 32;
    bool idled = false, pend = false;      // pend: the first warp wrote since the last barrier
    auto others = [&]() {
        if (!idled) idle();
        idled = true;
    };
    // Segments of consecutive narrow or wide waves {count | kind, first}.
    for (uint32_t sg = 0; sg < c.nfSeg; ++sg) {
        const uint2 S = __ldg(c.fSeg + sg);
        const uint32_t n = S.x & ~kSegKind;
        if (S.x & kSegNarrow) {
            pend = true;
            if (!w0) {
                others();
                continue;
            }
            const uint4* r = c.fLane + S.y + lane;
            uint4 next = __ldg(r);
            for (uint32_t w = 0; w < n; ++w) {
                const uint4 u = next;
                r += 32;
                if (w + 1 < n) next = __ldg(r);
                laneUpdate(M, u);
                __syncwarp();
            }
            continue;
        }
        if (pend) teamSync(t);
        pend = false;
        const uint32_t* ptr = c.fWavePtr + S.y;
        uint32_t b = ptr[0], e = ptr[1], e1 = ptr[min(2u, n)], k;
        bool two;
        auto mine = [&]() {
            two = c.fSplit && 2 * (e - b) <= t.nth;
            k = b + (two ? t.tid >> 1 : t.tid);
        };
        mine();
        ProgOp next;
        if (k < e) next = progOp(c.fW, k);
        for (uint32_t w = 0; w < n; ++w) {
            const uint32_t k0 = k, e0 = e;
            const bool two0 = two;
            ProgOp u = next;
            if (w + 1 < n) {
                b = e;
                e = e1;
                e1 = ptr[min(w + 3, n)];
                mine();
                if (k < e) next = progOp(c.fW, k);
            }
            if (two0) {
                if (k0 < e0) waveEntry(M, (t.tid & 1u) ? u.d.y : u.d.x, waveQuotient(M, u), u.off);
            } else {
                for (uint32_t j = k0; j < e0; j += t.nth) {
                    if (j != k0) u = progOp(c.fW, j);
                    const double q = waveQuotient(M, u);
                    waveEntry(M, u.d.x, q, u.off);
                    waveEntry(M, u.d.y, q, u.off);
                }
            }
            teamSync(t);
        }
    }
    double* S = c.runRows ? M + 2 * N + c.H : nullptr;
    if (!c.fWaves) forwardLevels(c, M, t, S);
    // back substitution: narrow levels and cable runs by the first warp
    for (uint32_t sg = 0; sg < c.nbSeg; ++sg) {
        const uint2 sgm = __ldg(c.bSeg + sg);
        const uint32_t n = sgm.x & ~kSegKind;
        if (sgm.x & kSegKind) {
            pend = true;
            if (!w0) {
                others();
                continue;
            }
            if (sgm.x & kSegRun) {
                const double* off = c.M + 2 * N + c.H;
                if (S && n >= kWarpRun) backwardWarpRun(M, off, N, sgm.y, n, S);
                else if (t.tid == 0) backwardCableRun(M, off, M + N, N, sgm.y, n);
                __syncwarp();
                continue;
            }
            uint32_t k = sgm.y + lane;
            ProgOp next = progOp(c.bLane, k);
            for (uint32_t l = 0; l < n; ++l, k += 32) {
                const ProgOp r = next;
                if (l + 1 < n) next = progOp(c.bLane, k + 32);
                if ((r.d.x & 0xFFFFu) != kNoIndex) substitute(c, M, c.bLane, k, r);
                __syncwarp();
            }
            continue;
        }
        if (pend) teamSync(t);
        pend = false;
        const uint32_t* ptr = c.bLevelPtr + sgm.y;
        uint32_t e = ptr[1], e1 = ptr[min(2u, n)], k = ptr[0] + t.tid;
        ProgOp next;
        if (k < e) next = progOp(c.bW, k);
        for (uint32_t l = 0; l < n; ++l) {
            const uint32_t k0 = k, e0 = e;
            const ProgOp r = next;
            if (l + 1 < n) {
                k = e + t.tid;
                e = e1;
                e1 = ptr[min(l + 3, n)];
                if (k < e) next = progOp(c.bW, k);
            }
            if (k0 < e0) substitute(c, M, c.bW, k0, r);
            for (uint32_t j = k0 + t.nth; j < e0; j += t.nth) substitute(c, M, c.bW, j, progOp(c.bW, j));
            teamSync(t);
        }
    }
    if (pend) teamSync(t);
}

// The same sweeps in global memory by one CTA, for a cell whose matrix does
// not fit in shared memory (above ~5,000 branched compartments).
__device__ __forceinline__ void waveUpdate(const DevCell& c, double* M, uint32_t k) {
    const int4 x = c.fWaveOps[2 * k], y = c.fWaveOps[2 * k + 1];
    const double q = quotient(M[y.x], M[y.y]);
    M[x.x] -= q * M[x.y];
    if (x.z >= 0) M[x.z] -= q * M[x.w];
}

__device__ __forceinline__ void backRowGlobal(const DevCell& c, const double* M, uint32_t k) {
    const uint32_t N = c.N, i = c.bRows[k];
    double v = M[N + i];
    for (uint32_t t = c.bTermPtr[k]; t < c.bTermPtr[k + 1]; ++t) {
        int2 term = c.bTerms[t];
        v -= M[term.x] * c.VMid[term.y];
    }
    c.VMid[i] = quotient(v, M[i]);
}

__device__ void eliminateGlobal(const DevCell& c, const Team& t) {
    double* M = c.M;
    const uint32_t N = c.N;
    const double* off = M + 2 * N + c.H;
    for (uint32_t w = 0; w < c.fWaves; ++w) {
        for (uint32_t k = c.fWavePtr[w] + t.tid; k < c.fWavePtr[w + 1]; k += t.nth) waveUpdate(c, M, k);
        teamSync(t);
    }
    if (!c.fWaves) forwardLevels(c, M, t, nullptr);
    for (uint32_t l = 0; l < c.bLevels; ++l) {
        if (const uint32_t run = c.bRun[l]) {
            if (t.tid == 0) backwardCableRun(M, off, c.VMid, N, c.bRunRow[l], run);
            l += run - 1;
        } else {
            for (uint32_t k = c.bLevelPtr[l] + t.tid; k < c.bLevelPtr[l + 1]; k += t.nth) backRowGlobal(c, M, k);
        }
        teamSync(t);
    }
}

// Of a cell stepped by a cluster, still in global memory: a forward wave or a
// back-substitution level of at least kClusterWide updates or rows is
// shared by all the cluster's CTAs, a cluster barrier after it (and before
// it, when rank 0 wrote alone since the last one); narrower ones are
// walked by rank 0's CTA with a CTA barrier.  The
// updates of a wave, and the rows of a level, are independent, so which
// thread of which CTA does one changes nothing: bit-identical.  Every CTA
// takes the same branches (they depend on the sizes
// alone), so all meet at every cluster barrier.  (One GB300, 8 CTAs, against
// rank 0 alone in global memory: 10,000 compartments 631 -> 498 us per step.)
constexpr uint32_t kClusterWide = 1024;

__device__ void eliminateGlobalCluster(const DevCell& c, cooperative_groups::cluster_group& cl, uint32_t rank,
                                       const Team& t, uint32_t g, uint32_t G) {
    if (!c.fWaves) {
        if (rank == 0) eliminateGlobal(c, t);
        return;
    }
    double* M = c.M;
    bool alone = false;      // rank 0 wrote since the last cluster barrier
    for (uint32_t w = 0; w < c.fWaves; ++w) {
        const uint32_t b0 = c.fWavePtr[w], e = c.fWavePtr[w + 1];
        if (e - b0 >= kClusterWide) {
            if (alone) cl.sync();
            alone = false;
            for (uint32_t k = b0 + g; k < e; k += G) waveUpdate(c, M, k);
            cl.sync();
        } else {
            if (rank == 0) {
                for (uint32_t k = b0 + t.tid; k < e; k += t.nth) waveUpdate(c, M, k);
                teamSync(t);
            }
            alone = true;
        }
    }
    const uint32_t N = c.N;
    for (uint32_t l = 0; l < c.bLevels; ++l) {
        if (const uint32_t run = c.bRun[l]) {
            if (rank == 0) {
                if (t.tid == 0) backwardCableRun(M, M + 2 * N + c.H, c.VMid, N, c.bRunRow[l], run);
                teamSync(t);
            }
            alone = true;
            l += run - 1;
            continue;
        }
        const uint32_t b0 = c.bLevelPtr[l], e = c.bLevelPtr[l + 1];
        if (e - b0 >= kClusterWide) {
            if (alone) cl.sync();
            alone = false;
            for (uint32_t k = b0 + g; k < e; k += G) backRowGlobal(c, M, k);
            cl.sync();
        } else {
            if (rank == 0) {
                for (uint32_t k = b0 + t.tid; k < e; k += t.nth) backRowGlobal(c, M, k);
                teamSync(t);
            }
            alone = true;
        }
    }
}

// ---- outputs of a step ---------------------------------------------------------
// SpikeGens (one thread), with V and Ca at the end of step `step`.
__device__ __forceinline__ void spikeGens(const DevCell& c, unsigned long long step, uint32_t& nSpikes) {
    const double currTime = c.dt * (double)(step + 1);
    for (uint32_t k = 0; k < c.SG; ++k) {
        if (lessThan(c.sgThreshold[k], c.V[c.sgCompt[k]])) {
            if (atMost(c.sgLast[k] + c.sgRefract[k], currTime + c.dt / 2.0) && !(c.sgEdge[k] && c.sgFired[k])) {
                if (nSpikes < c.spikeCap) {
                    c.spikeGen[nSpikes] = k;
                    c.spikeTime[nSpikes] = currTime;
                }
                ++nSpikes;
                c.sgLast[k] = currTime;
                c.sgFired[k] = 1;
            }
        } else {
            c.sgFired[k] = 0;
        }
    }
}

__device__ __forceinline__ void stimulus(const DevCell& c, unsigned long long step, uint32_t& stimPtr) {
    while (stimPtr < c.nStim && c.stimStep[stimPtr] <= step) {
        uint32_t h = c.stimCompt[stimPtr];
        c.injPresent[h] = 1;
        c.injBasal[h] = c.stimValue[stimPtr];
        ++stimPtr;
    }
}

// What the tick-4 objects of compartment ic are sent (HSolveActive::sendValues).
__device__ __forceinline__ void sendCompt(const DevCell& c, uint32_t k) {
    c.c2dVm[k] = c.V[c.c2dCompt[k]];
    if (c.c2dConc1[k] >= 0) c.c2dC1[k] = c.ca[c.c2dConc1[k]];
    if (c.c2dConc2[k] >= 0) c.c2dC2[k] = c.ca[c.c2dConc2[k]];
}

// One cell, `nsteps` steps, by team `t` or, with CL, by the cluster whose
// rank `rank` CTA this is.  Object k goes to thread k of the G threads
// (this one is g).  The matrix Mr is in shared memory (`own`; of a cluster in
// rank 0's, which the others reach through distributed shared memory) or,
// unless `shared`, the cell's in global memory.
// Fused steps (c.local: every pool and HHChannel2D reads and feeds its own
// compartment; no tick-1 objects, no recorded Gk or Ik): the end of a
// compartment's step (V, pools), its HHChannel2Ds and its next row are one
// pass of one thread, so a step has two barriers besides the elimination's;
// the outputs of a step, and the next step's SynChans and stimulus, which
// need nothing that the elimination writes, run while it does.
// Otherwise the phases run one after the other.
template <bool CL>
__device__ __forceinline__ void stepCell(const DevCell& c, uint32_t nsteps, const Team& t, bool shared, double* own,
                                         double* Mr, uint32_t rank, uint32_t g, uint32_t G) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    auto phase = [&]() {
        if (CL) cl.sync();
        else teamSync(t);
    };
    const uint32_t N = c.N;
    const double hdt = c.dt / 2.0;
    const bool fused = c.local && !c.nDif && !(c.nRec && c.recChan);
    const bool aux = g == (G > 32 ? G - 32 : 0);      // stimulus and SpikeGens: a thread of the last warp
    double* VMid = shared ? Mr + N : c.VMid;
    unsigned long long step = c.ctl->nSteps;
    uint32_t stimPtr = c.ctl->stimPtr, nSpikes = c.ctl->nSpikes, nSamples = c.ctl->nSamples;
    phase();
    auto record = [&](unsigned long long st) {
        if (c.nRec && ((st + 1) % c.recStride) == 0) {
            if (nSamples < c.recCap)
                for (uint32_t r = g; r < c.nRec; r += G)
                    c.recBuf[(size_t)nSamples * c.recLd + r] = recValue(c, c.recCompt[r]);
            ++nSamples;
        }
    };
    for (uint32_t s = 0; s < nsteps; ++s, ++step) {
        const bool first = s == 0, last = s + 1 == nsteps;
        if (first || !fused) {
            const double currTime = c.dt * (double)(step + 1);   // Clock: dt_ * endStep
            if (aux) stimulus(c, step, stimPtr);
            if (g == 0 && c.nDif) difProcess(c);                  // tick 1, before the gates read extCa
            for (uint32_t k = g; k < c.S; k += G) synchanStep(c, k, currTime);
            if (!fused)
                for (uint32_t k = g; k < c.K2; k += G) chan2dStep(c, k, c.c2dVm[k], c.c2dC1[k], c.c2dC2[k]);
            phase();
        }
        for (uint32_t h = g; h < c.H; h += G) Mr[2 * N + h] = c.HJ0[h];
        for (uint32_t ic = g; ic < N; ic += G) {
            if (fused && !first) finishCompt(c, ic, VMid, s == 1);
            rowStep(c, ic, hdt, fused, first, last, Mr);
        }
        phase();
        auto aside = [&](uint32_t a, uint32_t nA) {
            if (!fused) return;
            if (!first && aux) spikeGens(c, step - 1, nSpikes);
            if (last) return;
            if (aux) stimulus(c, step + 1, stimPtr);
            const double nextTime = c.dt * (double)(step + 2);
            for (uint32_t k = a; k < c.S; k += nA) synchanStep(c, k, nextTime);
        };
        if (fused && !first) record(step - 1);
        if (!shared) {
            aside(g, G);
            if (CL) eliminateGlobalCluster(c, cl, rank, t, g, G);
            else eliminateGlobal(c, t);
        } else if (CL) {
            if (rank) aside((rank - 1) * t.nth + t.tid, G - t.nth);
            else eliminateShared(c, own, t, [&]() {});
        } else if (t.nth > 32) {
            eliminateShared(c, own, t, [&]() { aside(t.tid - 32, t.nth - 32); });
        } else {
            aside(g, G);
            eliminateShared(c, own, t, [&]() {});
        }
        if (CL || !shared) phase();
        if (!fused) {
            for (uint32_t ic = g; ic < N; ic += G) c.V[ic] = __fma_rn(2.0, VMid[ic], -c.V[ic]);
            phase();
            for (uint32_t p = g; p < c.P; p += G) poolStep(c, p, VMid, first);
            phase();
            if (g == 0 && c.nDif) difSendIk(c);
            for (uint32_t k = g; k < c.K2; k += G) sendCompt(c, k);
            if (aux) spikeGens(c, step, nSpikes);
            record(step);
            phase();
        }
    }
    if (fused && nsteps) {
        for (uint32_t ic = g; ic < N; ic += G) finishCompt(c, ic, VMid, nsteps == 1);
        phase();
        for (uint32_t k = g; k < c.K2; k += G) sendCompt(c, k);
        if (aux) spikeGens(c, step - 1, nSpikes);
        record(step - 1);
    }
    if (aux) {
        c.ctl->nSteps = step;
        c.ctl->stimPtr = stimPtr;
        c.ctl->nSpikes = nSpikes;
        c.ctl->nSamples = nSamples;
    }
}

// The drop-in, one CTA.  `words`: the matrix is in shared memory (that many
// doubles), 0: in global memory.
__global__ void __launch_bounds__(512, 1) hsStepFp64(DevCell c, uint32_t words, uint32_t nsteps) {
    extern __shared__ double sMatrix[];
    const Team t{threadIdx.x, blockDim.x, 0};
    stepCell<false>(c, nsteps, t, words != 0, sMatrix, words ? sMatrix : c.M, 0, t.tid, t.nth);
}

// One cell stepped by a thread-block cluster.  On one SM a large cell's step
// is bound by the FP64 work of its channels and matrix rows (one SM's FP64
// pipe); the cluster's CTAs share that work -- object k goes to thread k of
// the cluster -- and write the rows into rank 0's shared memory, whose CTA
// eliminates.  Every object's arithmetic is unchanged and the phases keep
// their order, so the results are bit-identical to one CTA's.  The hardware
// cluster barrier (release/acquire at cluster scope) orders the phases.
__device__ __forceinline__ void stepCellCluster(const DevCell& c, uint32_t words, uint32_t nsteps, double* sm) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const Team t{threadIdx.x, blockDim.x, 0};
    const uint32_t rank = cl.block_rank();
    // warps of the cluster in turn over its CTAs: a few warps of objects
    // reach as many sub-partitions as there are
    const uint32_t nb = cl.num_blocks(), g = ((t.tid >> 5) * nb + rank) * 32 + (t.tid & 31u);
    stepCell<true>(c, nsteps, t, words != 0, sm, words ? cl.map_shared_rank(sm, 0) : c.M, rank, g, nb * t.nth);
    if (words) cl.sync();        // rank 0's shared memory outlives every access
}

__global__ void __launch_bounds__(256, 1) hsStepFp64Cluster(DevCell c, uint32_t words, uint32_t nsteps) {
    extern __shared__ double sMatrix[];
    stepCellCluster(c, words, nsteps, sMatrix);
}

// The cell descriptions are read from shared memory: a pointer per array, used
// all through the step.
__device__ __forceinline__ void copyCell(DevCell* dst, const DevCell* src, uint32_t tid, uint32_t nth) {
    const uint32_t n = sizeof(DevCell) / 8;
    const unsigned long long* a = reinterpret_cast<const unsigned long long*>(src);
    unsigned long long* b = reinterpret_cast<unsigned long long*>(dst);
    for (uint32_t i = tid; i < n; i += nth) b[i] = a[i];
}
static_assert(sizeof(DevCell) % 8 == 0, "DevCell is copied in 8-byte words");

// Separate drop-in solvers stepped in one launch (hs_process_group): CTA k
// steps solver k exactly as hsStepFp64 steps it alone; in the cluster form
// cluster k steps solver k exactly as hsStepFp64Cluster does.  `words`: doubles
// of shared memory a CTA has for its matrix.
__global__ void __launch_bounds__(256, 2) hsGroupStepFp64(const DevCell* __restrict__ cells, uint32_t words,
                                                          uint32_t nsteps) {
    extern __shared__ double sMatrix[];
    __shared__ DevCell c;
    copyCell(&c, cells + blockIdx.x, threadIdx.x, blockDim.x);
    __syncthreads();
    const Team t{threadIdx.x, blockDim.x, 0};
    const bool shared = c.smWords && c.smWords <= words;
    stepCell<false>(c, nsteps, t, shared, sMatrix, shared ? sMatrix : c.M, 0, t.tid, t.nth);
}

__global__ void __launch_bounds__(256, 2) hsGroupStepFp64Cluster(const DevCell* __restrict__ cells, uint32_t words,
                                                              uint32_t nsteps) {
    extern __shared__ double sMatrix[];
    __shared__ DevCell c;
    copyCell(&c, cells + blockIdx.x / cooperative_groups::this_cluster().num_blocks(), threadIdx.x, blockDim.x);
    __syncthreads();
    stepCellCluster(c, c.smWords <= words ? c.smWords : 0, nsteps, sMatrix);
}

// Batched FP64: one CTA per SM, in teams of `teamThreads` threads.  The CTA
// steps the cells of its own list (wholePtr) one after the other with all its
// threads, as the drop-in steps one cell; then each team steps its list
// (teamPtr), so that the elimination's latency of one cell overlaps the FP64
// work of the others.  Both forms do the drop-in's arithmetic in its order:
// results are bit-identical whichever form steps a cell.  `words`: doubles of
// shared memory for a whole-CTA cell's matrix; a team has its share.
__global__ void __launch_bounds__(512, 1) hsBatchStepFp64(const DevCell* __restrict__ cells,
                                                          const uint32_t* __restrict__ wholePtr,
                                                          const uint32_t* __restrict__ wholeCells,
                                                          const uint32_t* __restrict__ teamPtr,
                                                          const uint32_t* __restrict__ teamCells,
                                                          uint32_t teamThreads, uint32_t words, uint32_t nsteps) {
    extern __shared__ double sm[];
    const uint32_t nTeams = blockDim.x / teamThreads, team = threadIdx.x / teamThreads;
    DevCell* sCells = reinterpret_cast<DevCell*>(sm);
    double* sMatrix = sm + nTeams * (sizeof(DevCell) / 8);
    const uint32_t n0 = wholePtr[blockIdx.x + 1] - wholePtr[blockIdx.x];
    const uint32_t t0 = blockIdx.x * nTeams + team;
    const uint32_t n1 = teamPtr[t0 + 1] - teamPtr[t0];
    const uint32_t share = words / nTeams;
    for (uint32_t k = 0;; ++k) {
        if (k == n0 && n0) __syncthreads();     // the whole CTA's last cell is done everywhere
        if (k >= n0 + n1) break;
        const bool whole = k < n0;
        const Team t{whole ? threadIdx.x : threadIdx.x - team * teamThreads, whole ? blockDim.x : teamThreads,
                     whole ? 0 : team};
        const uint32_t cell = whole ? wholeCells[wholePtr[blockIdx.x] + k] : teamCells[teamPtr[t0] + k - n0];
        DevCell* c = sCells + (whole ? 0 : team);
        teamSync(t);                            // the team's last cell is done
        copyCell(c, cells + cell, t.tid, t.nth);
        teamSync(t);
        const uint32_t room = whole ? words : share;
        const bool shared = c->smWords && c->smWords <= room;
        double* M = sMatrix + (whole ? 0 : team * share);
        stepCell<false>(*c, nsteps, t, shared, M, shared ? M : c->M, 0, t.tid, t.nth);
    }
}

__device__ void reinitGatesCompt(const DevCell& c, uint32_t ic) {
    const Row vRow = tableRow(c.V[ic], c.vMin, c.vMax, c.vDx, c.vRdx, c.vRows);
    for (uint32_t q = c.chanPtr[ic]; q < c.chanPtr[ic + 1]; ++q) {
        const uint4 A = c.chanA[q];
        uint32_t s = A.y;
        double C1, C2;
        if (A.x & 0xFu) {
            tableLookup(c.vTab, c.vCol, (int32_t)A.z, vRow, C1, C2);
            c.state[s++] = C1 / C2;
        }
        if (A.x & 0xF0u) {
            tableLookup(c.vTab, c.vCol, (int32_t)A.w, vRow, C1, C2);
            c.state[s++] = C1 / C2;
        }
        if (A.x & 0xF00u) {
            const int32_t src = c.zSrc[q];
            const double ca = src >= 0 ? c.ca[src] : c.extCa[q];
            if (src >= 0 || ca > 0) {
                const Row r = tableRow(ca, c.caMin, c.caMax, c.caDx, c.caRdx, c.caRows);
                tableLookup(c.caTab, c.caCol, c.colZ[q], r, C1, C2);
            } else {
                tableLookup(c.vTab, c.vCol, c.colZ[q], vRow, C1, C2);
            }
            c.state[s] = C1 / C2;
        }
    }
}

// HSolveActive::reinit (hsolve/HSolveActiveSetup.cpp:43-160) and the reinit
// of the tick-1/4 objects (SynChan::vReinit, SimpleSynHandler::vReinit with
// the description's events queued again, HHChannel2D X), one warp per cell.
__global__ void hsReinitFp64(const DevCell* __restrict__ cells, uint32_t nCells) {
    uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t lane = threadIdx.x & 31;
    if (w >= nCells) return;
    const DevCell& c = cells[w];
    for (uint32_t k = lane; k < c.S; k += 32) {
        c.synXc1[k] = c.synConst[5 * k];
        c.synXc2[k] = c.synConst[5 * k + 1];
        c.synYc1[k] = c.synConst[5 * k + 2];
        c.synYc2[k] = c.synConst[5 * k + 3];
        c.synNorm[k] = c.synConst[5 * k + 4];
        c.synX[k] = 0.0;
        c.synY[k] = 0.0;
        c.synAct[k] = 0.0;
        c.synGk[k] = 0.0;
        c.evCur[k] = c.evPtr[k];
    }
    for (uint32_t i = lane; i < c.N; i += 32) {
        c.V[i] = c.initVm[i];
        c.ext[2 * i] = 0.0;
        c.ext[2 * i + 1] = 0.0;
        c.injVarying[i] = 0.0;
    }
    for (uint32_t k = lane; k < c.SG; k += 32) c.sgLast[k] = -c.sgRefract[k];
    for (uint32_t p = lane; p < c.P; p += 32) {
        c.iCa[p] = 0.0;
        c.c[p] = 0.0;
        c.ca[p] = c.CaBasal[p];
    }
    if (lane == 0) {
        c.ctl->nSteps = 0;
        c.ctl->stimPtr = 0;
        c.ctl->nSpikes = 0;
        c.ctl->nSamples = 0;
        c.ctl->err = 0;
    }
    __syncwarp();
    // sendValues: the tick-4 objects see initVm and CaBasal
    // tick-1 objects reinit before the solver: their concentrations reach
    // the channels' external calcium the gates start from
    if (lane == 0 && c.nDif) difReinit(c);
    __syncwarp();
    for (uint32_t k = lane; k < c.K2; k += 32) {
        c.c2dX[k] = c.c2dX0[k];
        c.c2dGk[k] = 0.0;
        c.c2dVm[k] = c.V[c.c2dCompt[k]];
        c.c2dC1[k] = c.c2dConc1[k] >= 0 ? c.ca[c.c2dConc1[k]] : 0.0;
        c.c2dC2[k] = c.c2dConc2[k] >= 0 ? c.ca[c.c2dConc2[k]] : 0.0;
    }
    for (uint32_t ic = lane; ic < c.N; ic += 32) reinitGatesCompt(c, ic);
    // a Table reading Vm at reinit records sample 0
    if (c.nRec && c.recCap) {
        for (uint32_t r = lane; r < c.nRec; r += 32) c.recBuf[r] = recValue(c, c.recCompt[r]);
        __syncwarp();
        if (lane == 0) c.ctl->nSamples = 1;
    }
}

__global__ void hsScatterFields(const FieldWrite* __restrict__ w, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const FieldWrite x = w[i];
    if (x.size == 8) *static_cast<unsigned long long*>(x.addr) = x.bits;
    else if (x.size == 4) *static_cast<uint32_t*>(x.addr) = (uint32_t)x.bits;
    else *static_cast<uint8_t*>(x.addr) = (uint8_t)x.bits;
}

// Spike read-back of a batch: each cell's spike count, then every cell's
// stored spikes gathered into one list (cell c at off[c] .. off[c+1]), so
// that the host reads all cells with one copy per array.
__global__ void hsSpikeCountsFp64(const DevCell* __restrict__ cells, uint32_t nCells, uint32_t* __restrict__ counts) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < nCells) counts[c] = cells[c].ctl->nSpikes;
}

__global__ void hsGatherSpikesFp64(const DevCell* __restrict__ cells, uint32_t nCells,
                                   const uint32_t* __restrict__ off, uint32_t* __restrict__ gen,
                                   double* __restrict__ time) {
    const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (c >= nCells) return;
    const uint32_t o = off[c], m = off[c + 1] - o;
    const DevCell& d = cells[c];
    for (uint32_t i = lane; i < m; i += 32) {
        gen[o + i] = d.spikeGen[i];
        time[o + i] = d.spikeTime[i];
    }
}

__global__ void hsGatherSpikesMixed(const uint32_t* __restrict__ srcGen, const float* __restrict__ srcTime,
                                    uint32_t cap, uint32_t nCells, const uint32_t* __restrict__ off,
                                    uint32_t* __restrict__ gen, double* __restrict__ time) {
    const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (c >= nCells) return;
    const uint32_t o = off[c], m = off[c + 1] - o;
    for (uint32_t i = lane; i < m; i += 32) {
        gen[o + i] = srcGen[(size_t)c * cap + i];
        time[o + i] = (double)srcTime[(size_t)c * cap + i];
    }
}

// One value per entry of a gather list: out[k] = *src[k] (a double, or a
// float when f32), NaN for a null entry.
__global__ void hsGatherValues(const void* const* __restrict__ src, uint32_t f32, uint64_t n,
                               double* __restrict__ out) {
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const void* p = src[k];
    out[k] = !p ? __longlong_as_double(0x7FF8000000000000ll)
                : f32 ? (double)*static_cast<const float*>(p) : *static_cast<const double*>(p);
}

cudaError_t launchGatherValues(const void* const* src, uint32_t f32, uint64_t n, double* out, cudaStream_t st) {
    if (!n) return cudaSuccess;
    hsGatherValues<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(src, f32, n, out);
    return cudaGetLastError();
}

cudaError_t launchSpikeCountsFp64(const DevCell* cells, uint32_t nCells, uint32_t* counts, cudaStream_t st) {
    if (!nCells) return cudaSuccess;
    hsSpikeCountsFp64<<<(nCells + 255) / 256, 256, 0, st>>>(cells, nCells, counts);
    return cudaGetLastError();
}

cudaError_t launchGatherSpikes(const DevCell* cells, const uint32_t* srcGen, const float* srcTime, uint32_t cap,
                               uint32_t nCells, const uint32_t* off, uint32_t* gen, double* time,
                               cudaStream_t st) {
    if (!nCells) return cudaSuccess;
    const uint32_t blocks = (nCells * 32 + 255) / 256;
    if (cells) hsGatherSpikesFp64<<<blocks, 256, 0, st>>>(cells, nCells, off, gen, time);
    else hsGatherSpikesMixed<<<blocks, 256, 0, st>>>(srcGen, srcTime, cap, nCells, off, gen, time);
    return cudaGetLastError();
}

cudaError_t launchScatterFields(const FieldWrite* w, uint32_t n, cudaStream_t st) {
    if (!n) return cudaSuccess;
    hsScatterFields<<<(n + 255) / 256, 256, 0, st>>>(w, n);
    return cudaGetLastError();
}

namespace {

// Doubles of shared memory that a kernel with `statics` bytes of its own can
// have, on the current device.
uint32_t roomWords(size_t statics) {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    return (size_t)optin > statics ? (uint32_t)(((size_t)optin - statics) / 8) : 0;
}

cudaLaunchConfig_t clusterConfig(cudaLaunchAttribute* attr, uint32_t grid, uint32_t ctas, size_t smem,
                                 cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

uint32_t fp64MatrixRoom() { return roomWords(sizeof(DevCell)); }

cudaError_t launchStepFp64(const DevCell& c, uint32_t nsteps, cudaStream_t st) {
    const uint32_t words = c.smWords <= fp64MatrixRoom() ? c.smWords : 0;
    cudaError_t e = allowShared((const void*)hsStepFp64);
    if (e != cudaSuccess) return e;
    hsStepFp64<<<1, c.N > 256 ? 512 : 256, 8 * (size_t)words, st>>>(c, words, nsteps);
    return cudaGetLastError();
}

cudaError_t launchStepFp64Cluster(const DevCell& c, uint32_t ctas, uint32_t nsteps, cudaStream_t st) {
    const uint32_t words = c.smWords <= fp64MatrixRoom() ? c.smWords : 0;
    cudaError_t e = allowShared((const void*)hsStepFp64Cluster);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = clusterConfig(attr, ctas, ctas, 8 * (size_t)words, st);
    return cudaLaunchKernelEx(&cfg, hsStepFp64Cluster, c, words, nsteps);
}

// `ctas` CTAs per solver: 1 = one CTA each (no cluster), 2..8 = a cluster
// each; `words`: doubles of shared memory per CTA, the most that a member's
// matrix needs (members that need more use global memory)
cudaError_t launchGroupStepFp64(const DevCell* cells, uint32_t n, uint32_t ctas, uint32_t words, uint32_t nsteps,
                                cudaStream_t st) {
    if (!n) return cudaSuccess;
    const size_t smem = 8 * (size_t)words;
    if (ctas <= 1) {
        cudaError_t e = allowShared((const void*)hsGroupStepFp64);
        if (e != cudaSuccess) return e;
        hsGroupStepFp64<<<n, 256, smem, st>>>(cells, words, nsteps);
        return cudaGetLastError();
    }
    cudaError_t e = allowShared((const void*)hsGroupStepFp64Cluster);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = clusterConfig(attr, n * ctas, ctas, smem, st);
    return cudaLaunchKernelEx(&cfg, hsGroupStepFp64Cluster, cells, words, nsteps);
}

// Doubles of shared memory that the FP64 batch's CTA of `teams` teams has for
// matrices.
uint32_t fp64BatchWords(uint32_t teams) { return roomWords(teams * sizeof(DevCell)); }

cudaError_t launchBatchStepFp64(const DevCell* cells, const uint32_t* wholePtr, const uint32_t* wholeCells,
                                const uint32_t* teamPtr, const uint32_t* teamCells, uint32_t nBlocks,
                                uint32_t teams, uint32_t teamThreads, uint32_t words, uint32_t nsteps,
                                cudaStream_t st) {
    const size_t smem = teams * sizeof(DevCell) + 8 * (size_t)words;
    cudaError_t e = allowShared((const void*)hsBatchStepFp64);
    if (e != cudaSuccess) return e;
    hsBatchStepFp64<<<nBlocks, teams * teamThreads, smem, st>>>(cells, wholePtr, wholeCells, teamPtr, teamCells,
                                                                teamThreads, words, nsteps);
    return cudaGetLastError();
}

cudaError_t launchReinitFp64(const DevCell* cells, uint32_t nCells, cudaStream_t st) {
    uint32_t blocks = (nCells * 32 + 255) / 256;
    hsReinitFp64<<<blocks ? blocks : 1, 256, 0, st>>>(cells, nCells);
    return cudaGetLastError();
}

}  // namespace hsg
