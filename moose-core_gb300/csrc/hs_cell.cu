// hs_cell.cu -- upload of a CellPlan into a device arena (see hs_cell.h).
#include <algorithm>
#include <cstring>

#include "hs_cell.h"

namespace hsg {

namespace {

// The arrays of a cell: small ones, and the zeros between them, are gathered on
// the host and sent together, larger ones by themselves.  A copy from
// pageable memory has a cost of its own, and a cell has about 90 arrays: a
// drop-in solver of 200 compartments is created in 0.97 ms, 1.06 with a copy
// for each.
struct Uploader {
    Arena& a;
    cudaStream_t st;
    std::vector<std::shared_ptr<void>>& sent;
    cudaError_t err = cudaSuccess;
    std::vector<char> part = {};       // bytes [first, first + part.size()) of the arena, to be sent
    size_t first = 0;
    static constexpr size_t kDirect = 64 << 10;
    // `v` outlives the copies, as the plan does
    template <class T>
    T* put(const std::vector<T>& v) {
        T* p = a.take<T>(v.empty() ? 1 : v.size());
        if (p) send(p, v);
        return p;
    }
    template <class T>
    void send(T* p, const std::vector<T>& v) {
        if (!v.empty() && err == cudaSuccess) add(reinterpret_cast<char*>(p) - a.base, v.data(), v.size() * sizeof(T));
    }
    template <class T>
    T* put(std::vector<T>&& v) {
        T* p = put(static_cast<const std::vector<T>&>(v));
        if (p && v.size() * sizeof(T) >= kDirect) keep(std::move(v));
        return p;
    }
    template <class T>
    T* zeros(size_t n) {
        return a.take<T>(n ? n : 1);    // the arena is memset to 0 before upload
    }
    const double* table(const Table& t) {
        if (a.base) return put(pairTable(t));
        const size_t n = t.nCol ? 2 * (size_t)(t.nPts - 1) * t.nCol : 0;    // pairTable's size
        return a.take<double>(n ? n : 1);
    }
    void add(size_t at, const void* src, size_t bytes) {
        if (bytes >= kDirect || part.empty() || at - first - part.size() >= kDirect) send();
        if (bytes >= kDirect) {
            err = cudaMemcpyAsync(a.base + at, src, bytes, cudaMemcpyHostToDevice, st);
            return;
        }
        if (part.empty()) first = at;
        part.resize(at - first, 0);
        part.insert(part.end(), static_cast<const char*>(src), static_cast<const char*>(src) + bytes);
    }
    cudaError_t send() {
        if (!part.empty() && err == cudaSuccess) {
            err = cudaMemcpyAsync(a.base + first, part.data(), part.size(), cudaMemcpyHostToDevice, st);
            keep(std::move(part));
        }
        part.clear();
        return err;
    }
    // (a moved vector's elements stay where they are)
    template <class T>
    void keep(std::vector<T>&& v) { sent.push_back(std::make_shared<std::vector<T>>(std::move(v))); }
};

}  // namespace

// Per row i and species {A_i, A_{i+1} - A_i, B_i, B_{i+1} - B_i}: the lookups
// interpolate between rows i and i + 1, and the last row is never the lower.
std::vector<double> pairTable(const Table& t) {
    std::vector<double> out(t.nCol ? 2 * (size_t)(t.nPts - 1) * t.nCol : 0);
    double* o = out.data();
    for (const double *a = t.data.data(), *end = a + out.size() / 2; a != end; ++a, o += 2) {
        o[0] = a[0];
        o[1] = a[t.nCol] - a[0];
    }
    return out;
}

namespace {

uint32_t powCode(double p) {
    if (!(p > 0.0)) return 0;
    for (uint32_t k = 1; k <= 4; ++k)
        if (p == (double)k) return k;
    return kPowGeneral;
}

// The sweeps' programs with 16-bit entries for a matrix in shared memory
// (DevCell::fW, bW, ...); false where they do not fit the encoding.
struct Compact {
    std::vector<uint4> fW, bW, fLane, bLane;
    std::vector<uint32_t> bX;
    std::vector<uint2> fSeg, bSeg;
    bool split = true, made = false;
};

bool compactPrograms(const CellPlan& P, Compact& C) {
    const uint32_t N = P.N, offBase = 2 * N + P.H, kNone = 0xFFFFu, kOff = 0xFFFEu;
    if (offBase >= kOff) return false;
    C.fW.reserve(2 * P.fWaveOps.size());
    C.bW.reserve(2 * P.bRows.size());
    C.fLane.reserve(32 * P.fWavePtr.size());
    C.bLane.reserve(64 * P.bLevelPtr.size());
    auto offOf = [&](uint32_t row) {
        uint64_t u = 0;
        if (row < N) std::memcpy(&u, &P.off[row], 8);
        return make_uint2((uint32_t)u, (uint32_t)(u >> 32));
    };
    for (const FwdPair& f : P.fWaveOps) {
        uint32_t row = 0xFFFFFFFFu, l = (uint32_t)f.l;
        if (l >= offBase) {
            row = l - offBase;
            l = kOff;
        }
        bool ok = true;
        auto entry = [&](int32_t a) {
            if ((uint32_t)a < offBase) return (uint32_t)a;
            ok = ok && (uint32_t)a - offBase == row;      // the update's own off-diagonal
            return kOff;
        };
        const uint32_t a1 = entry(f.a1), a2 = f.t2 >= 0 ? entry(f.a2) : 0u, t2 = f.t2 >= 0 ? (uint32_t)f.t2 : kNone;
        if (!ok) return false;
        const uint2 o = offOf(row);
        C.fW.push_back(make_uint4((uint32_t)f.t1 | a1 << 16, t2 | a2 << 16, l | (uint32_t)f.p << 16, 0));
        C.fW.push_back(make_uint4(o.x, o.y, 0, 0));
        if (f.t2 >= 0) {
            // two lanes may change an update's entries where neither reads
            // what the other writes
            for (int32_t r : {f.l, f.p, f.a1, f.a2})
                if (r == f.t1 || r == f.t2) C.split = false;
            if (f.t1 == f.t2) C.split = false;
        }
    }
    for (size_t k = 0; k < P.bRows.size(); ++k) {
        const uint32_t i = P.bRows[k], t0 = P.bTermPtr[k], n = P.bTermPtr[k + 1] - t0;
        if (n > 0xFFFFu) return false;
        uint32_t term[4] = {kNone, 0, 0, 0}, row = N;
        const uint32_t x0 = (uint32_t)C.bX.size();
        for (uint32_t t = 0; t < n; ++t) {
            const BwdTerm& x = P.bTerms[t0 + t];
            uint32_t co = (uint32_t)x.coef;
            if (co >= offBase) {
                if (t || co - offBase != i) return false;
                co = kOff;
                row = i;
            }
            const uint32_t w = co | (uint32_t)x.src << 16;
            if (t < 4) term[t] = w;
            else C.bX.push_back(w);
        }
        const uint2 o = offOf(row);
        C.bW.push_back(make_uint4(i | n << 16, term[0], term[1], term[2]));
        C.bW.push_back(make_uint4(o.x, o.y, term[3], x0));
    }
    auto grow = [](std::vector<uint2>& seg, uint32_t kind, uint32_t first) {
        if (!seg.empty() && (seg.back().x & kSegKind) == kind && kind != kSegRun) ++seg.back().x;
        else seg.push_back(make_uint2(1u | kind, first));
    };
    const uint32_t W = P.fWavePtr.empty() ? 0 : (uint32_t)P.fWavePtr.size() - 1;
    const uint4 idle = make_uint4(kNone, 0, 0, 0);
    for (uint32_t w = 0; w < W; ++w) {
        const uint32_t b = P.fWavePtr[w], n = P.fWavePtr[w + 1] - b;
        if (!C.split || n > 16) {
            grow(C.fSeg, 0, w);
            continue;
        }
        grow(C.fSeg, kSegNarrow, (uint32_t)C.fLane.size());
        for (uint32_t lane = 0; lane < 32; ++lane) {
            if (lane >= 2 * n) {
                C.fLane.push_back(idle);
                continue;
            }
            const uint4 d = C.fW[2 * (b + lane / 2)], o = C.fW[2 * (b + lane / 2) + 1];
            C.fLane.push_back(make_uint4(lane & 1 ? d.y : d.x, d.z, o.x, o.y));
        }
    }
    const uint32_t L = (uint32_t)P.bLevelPtr.size() - 1;
    for (uint32_t l = 0; l < L; ++l) {
        if (P.bRun[l]) {
            C.bSeg.push_back(make_uint2(P.bRun[l] | kSegRun, P.bRunRow[l]));
            l += P.bRun[l] - 1;
            continue;
        }
        const uint32_t b = P.bLevelPtr[l], n = P.bLevelPtr[l + 1] - b;
        if (n > 32) {
            grow(C.bSeg, 0, l);
            continue;
        }
        grow(C.bSeg, kSegNarrow, (uint32_t)C.bLane.size() / 2);
        for (uint32_t lane = 0; lane < 32; ++lane) {
            C.bLane.push_back(lane < n ? C.bW[2 * (b + lane)] : idle);
            C.bLane.push_back(lane < n ? C.bW[2 * (b + lane) + 1] : idle);
        }
    }
    return true;
}

}  // namespace

cudaError_t layoutCell(const CellPlan& P, Arena& a, DevCell& c, uint32_t spikeCap,
                       cudaStream_t st, CellUpload& up, const CellShared* sh, Arena* spikes) {
    Uploader u{a, st, up.sent};
    const uint32_t N = P.N, H = P.H;
    std::memset(&c, 0, sizeof(c));
    c.N = N; c.H = H; c.C = P.C; c.G = P.G; c.P = P.P; c.K2 = P.K2; c.S = P.S; c.SG = P.SG;
    c.nStim = (uint32_t)P.stimStep.size();
    c.fLevels = (uint32_t)P.fLevelPtr.size() - 1;
    c.bLevels = (uint32_t)P.bLevelPtr.size() - 1;
    c.caAdvance = 1;
    c.dt = P.dtSetup;
    c.V = u.put(P.V0);
    c.initVm = sh ? sh->initVm : u.put(P.initVm);
    c.synConst = sh ? sh->synConst : u.zeros<double>(5 * (size_t)P.S);
    c.c2dX0 = u.put(P.c2dX0);
    c.VMid = u.zeros<double>(N);
    {
        std::vector<double> M(3 * (size_t)N + H, 0.0);
        for (uint32_t h = 0; h < H; ++h) M[2 * N + h] = P.HJ0[h];
        for (uint32_t i = 0; i < N; ++i) M[2 * N + H + i] = P.off[i];
        c.M = u.put(std::move(M));
    }
    c.HJ0 = u.put(P.HJ0);
    c.HS2 = u.put(P.HS2);
    c.CmByDt = u.put(P.CmByDt);
    c.EmByRm = u.put(P.EmByRm);
    c.injBasal = u.put(P.injBasal);
    c.injVarying = u.zeros<double>(N);
    c.ext = u.zeros<double>(2 * (size_t)N);
    c.prevExt = u.zeros<double>(2 * (size_t)N);
    c.chanPtr = u.put(P.chanPtr);
    c.poolPtr = u.put(P.poolPtr);
    c.extPtr = u.put(P.extPtr);
    c.extList = u.put(P.extList);
    c.fWaves = P.fWavePtr.empty() ? 0 : (uint32_t)P.fWavePtr.size() - 1;
    if (!c.fWaves) {                // (with waves, nothing reads the forward level programs)
        c.fLevelPtr = u.put(P.fLevelPtr);
        c.fOpPtr = u.put(P.fOpPtr);
        c.fOps = reinterpret_cast<const int4*>(u.put(P.fOps));
        c.fRun = u.put(P.fRun);
        c.fRunRow = u.put(P.fRunRow);
    }
    c.bLevelPtr = u.put(P.bLevelPtr);
    c.bRows = u.put(P.bRows);
    c.bTermPtr = u.put(P.bTermPtr);
    c.bTerms = reinterpret_cast<const int2*>(u.put(P.bTerms));
    c.bRun = u.put(P.bRun);
    c.bRunRow = u.put(P.bRunRow);
    c.fWavePtr = u.put(P.fWavePtr);
    c.fWaveOps = reinterpret_cast<const int4*>(u.put(P.fWaveOps));
    {
        auto programs = std::static_pointer_cast<Compact>(up.programs);
        if (!programs) {
            programs = std::make_shared<Compact>();
            if (!compactPrograms(P, *programs)) *programs = Compact();
            else programs->made = true;
        }
        up.programs = a.base ? nullptr : programs;
        Compact& C = *programs;
        uint32_t longest = 0;      // runs walked as runs: forward only without waves
        for (uint32_t r : P.bRun) longest = std::max(longest, r);
        if (P.fWavePtr.empty())
            for (uint32_t r : P.fRun) longest = std::max(longest, r);
        c.runRows = longest >= kWarpRun ? longest : 0;
        c.smWords = C.made ? 2 * N + H + 2 * c.runRows : 0;
        c.fSplit = C.split;
        c.nfSeg = (uint32_t)C.fSeg.size();
        c.nbSeg = (uint32_t)C.bSeg.size();
        c.fW = u.put(C.fW);
        c.bW = u.put(C.bW);
        c.bX = u.put(C.bX);
        c.fLane = u.put(C.fLane);
        c.bLane = u.put(C.bLane);
        c.fSeg = u.put(C.fSeg);
        c.bSeg = u.put(C.bSeg);
        if (a.base) up.sent.push_back(programs);
    }
    c.Gbar = u.put(P.Gbar);
    c.Ek = u.put(P.Ek);
    c.Xpow = u.put(P.Xpow);
    c.Ypow = u.put(P.Ypow);
    c.Zpow = u.put(P.Zpow);
    c.mod = u.put(P.modulation);
    c.Gk = u.zeros<double>(P.C);
    c.state = u.put(P.state0);
    c.extCa = u.zeros<double>(P.C);
    c.instant = u.put(P.instant);
    {
        std::vector<uint4> ca(P.C);
        for (uint32_t q = 0; q < P.C; ++q)
            ca[q] = make_uint4(powCode(P.Xpow[q]) | powCode(P.Ypow[q]) << 4 | powCode(P.Zpow[q]) << 8,
                               (uint32_t)P.stateOff[q], (uint32_t)P.colX[q], (uint32_t)P.colY[q]);
        c.chanA = u.put(std::move(ca));
    }
    c.colZ = u.put(P.colZ);
    c.zSrc = u.put(P.zSrc);
    {
        std::vector<uint32_t> cc(P.C);
        for (uint32_t ic = 0; ic < N; ++ic)
            for (uint32_t q = P.chanPtr[ic]; q < P.chanPtr[ic + 1]; ++q) cc[q] = ic;
        std::vector<uint32_t> poolCompt(P.P);
        for (uint32_t ic = 0; ic < N; ++ic)
            for (uint32_t p = P.poolPtr[ic]; p < P.poolPtr[ic + 1]; ++p) poolCompt[p] = ic;
        bool local = true;
        for (uint32_t p = 0; p < P.P; ++p)
            for (uint32_t f = P.feedPtr[p]; f < P.feedPtr[p + 1]; ++f) local = local && cc[P.feedChan[f]] == poolCompt[p];
        for (uint32_t q = 0; q < P.C; ++q)
            local = local && (P.zSrc[q] < 0 || poolCompt[P.zSrc[q]] == cc[q]);
        for (uint32_t k = 0; k < P.K2; ++k)
            for (int32_t p : {P.c2dConc1[k], P.c2dConc2[k]}) local = local && (p < 0 || poolCompt[p] == P.c2dCompt[k]);
        c.local = local;
        c.chanCompt = u.put(std::move(cc));
    }
    c.c = u.put(P.c0);
    c.CaBasal = u.put(P.CaBasal);
    c.f1 = u.put(P.f1);
    c.f2 = u.put(P.f2);
    c.ceil = u.put(P.ceiling);
    c.floor_ = u.put(P.floor_);
    c.ca = u.zeros<double>(P.P);
    c.iCa = u.zeros<double>(P.P);
    c.feedPtr = u.put(P.feedPtr);
    c.feedChan = u.put(P.feedChan);
    c.vTab = sh ? sh->vTab : u.table(P.vTable);
    c.vCol = P.vTable.nCol; c.vMin = P.vTable.min; c.vMax = P.vTable.max; c.vDx = P.vTable.dx;
    c.vRows = P.vTable.nPts;
    c.vRdx = 1.0 / c.vDx;
    c.caTab = sh ? sh->caTab : u.table(P.caTable);
    c.caCol = P.caTable.nCol; c.caMin = P.caTable.min; c.caMax = P.caTable.max; c.caDx = P.caTable.dx;
    c.caRows = P.caTable.nPts;
    c.caRdx = 1.0 / c.caDx;
    {
        std::vector<double> geom;
        std::vector<uint64_t> off;
        std::vector<uint32_t> nn;
        size_t nAB = 0;
        for (const Gate2D& g : P.gates2d) {
            off.push_back(nAB);
            nAB += g.AB.size();
            geom.insert(geom.end(), {g.xmin, g.xmax, g.ymin, g.ymax, g.invDx, g.invDy});
            nn.push_back(g.nx);
            nn.push_back(g.ny);
        }
        if (sh) {
            c.g2dAB = sh->g2dBase;
            c.g2dOff = u.put(sh->g2dOff);
        } else {
            double* AB = a.take<double>(nAB ? nAB : 1);
            c.g2dAB = AB;
            for (size_t g = 0; AB && g < off.size(); ++g) u.send(AB + off[g], P.gates2d[g].AB);
            c.g2dOff = u.put(std::move(off));
        }
        c.g2dGeom = u.put(std::move(geom));
        c.g2dN = u.put(std::move(nn));
    }
    c.c2dCompt = u.put(P.c2dCompt);
    c.c2dGate = u.put(P.c2dGate);
    {
        auto dep = [](int32_t d) { return d < 0 || d > 2 ? 3u : (uint32_t)d; };
        std::vector<uint32_t> ka(P.K2);
        for (uint32_t k = 0; k < P.K2; ++k)
            ka[k] = powCode(P.c2dXpow[k]) | dep(P.c2dDep0[k]) << 4 | dep(P.c2dDep1[k]) << 8 |
                    ((uint32_t)P.c2dInstant[k] & 0xFu) << 12;
        c.c2dA = u.put(std::move(ka));
    }
    c.c2dConc1 = u.put(P.c2dConc1);
    c.c2dConc2 = u.put(P.c2dConc2);
    c.c2dGbar = u.put(P.c2dGbar);
    c.c2dEk = u.put(P.c2dEk);
    c.c2dXpow = u.put(P.c2dXpow);
    c.c2dMod = u.put(P.c2dMod);
    c.c2dX = u.put(P.c2dX0);
    c.c2dGk = u.zeros<double>(P.K2);
    c.c2dVm = u.zeros<double>(P.K2);
    c.c2dC1 = u.zeros<double>(P.K2);
    c.c2dC2 = u.zeros<double>(P.K2);
    c.synEk = u.put(P.synEk);
    c.synMod = u.put(P.synMod);
    c.synX = u.zeros<double>(P.S);
    c.synY = u.zeros<double>(P.S);
    c.synAct = u.zeros<double>(P.S);
    c.synGk = u.zeros<double>(P.S);
    c.synXc1 = u.zeros<double>(P.S);
    c.synXc2 = u.zeros<double>(P.S);
    c.synYc1 = u.zeros<double>(P.S);
    c.synYc2 = u.zeros<double>(P.S);
    c.synNorm = u.zeros<double>(P.S);
    c.evPtr = u.put(P.evPtr);
    c.evCur = u.put(P.evPtr);
    c.evTime = u.put(P.evTime);
    c.evW = u.put(P.evW);
    c.sgCompt = u.put(P.sgCompt);
    c.sgThreshold = u.put(P.sgThreshold);
    c.sgRefract = u.put(P.sgRefract);
    c.sgLast = u.zeros<double>(P.SG);
    c.sgEdge = u.put(P.sgEdge);
    c.sgFired = u.zeros<int32_t>(P.SG);
    c.spikeCap = spikeCap;
    Arena& sa = spikes ? *spikes : a;
    c.spikeGen = sa.take<uint32_t>(spikeCap);
    c.spikeTime = sa.take<double>(spikeCap);
    c.stimStep = u.put(P.stimStep);
    c.stimCompt = u.put(P.stimCompt);
    c.stimValue = u.put(P.stimValue);
    c.injPresent = u.put(P.injPresent);
    c.nDif = P.nDif;
    if (P.nDif) {
        c.difKind = u.put(P.difKind);
        c.difPar = u.put(P.difPar);
        c.difOff = u.put(P.difOff);
        c.difDst = u.put(P.difDst);
        c.ikOff = u.put(P.ikOff);
        c.ikDst = u.put(P.ikDst);
        // state; a DifBuffer starts from its activation field
        std::vector<double> st((size_t)kDifState * P.nDif, 0.0);
        for (uint32_t k = 0; k < P.nDif; ++k)
            if (P.difKind[k] == HS_DIF_BUFFER) st[9 * (size_t)P.nDif + k] = P.difPar[(size_t)k * HS_DIF_NPAR + 11];
        c.difState = u.put(std::move(st));
    }
    c.nRec = 0;
    c.recStride = 1;
    c.recCap = 0;
    c.recLd = 0;
    c.ctl = u.zeros<DevCtl>(1);
    return u.send();
}

void synConsts(const CellPlan& P, double dt, double* out) {
    for (uint32_t k = 0; k < P.S; ++k)
        synchanConstants(P.synTau1[k], P.synTau2[k], P.synGbar[k], dt, out + 5 * k, out + 5 * k + 1,
                         out + 5 * k + 2, out + 5 * k + 3, out + 5 * k + 4);
}

}  // namespace hsg
