// Device-side views of the GAMERA Model/Grid/State/Solver data, shared by
// every build variant of the step kernels and by the C ABI.
#pragma once
#include <cuda.h>
#include "gam_layout.cuh"

// Solar-wind boundary data (apps/wind.F90:206-391) for a constant wind: the
// blend weights and wind face fluxes depend only on the grid and the wind
// direction, so they are computed once on the host (libm acos/exp, the same
// expressions as wgtWind/RampDown) and stored for the 4 ghost layers:
// entry (n-1) + 4*(j + (Nj+1)*k) for ghost layer n = 1..4.
struct WindData {
    double state[8];    // rho, P, Vx, Vy, Vz, Bx, By, Bz
    const double* wC;   // weight at the ghost cell centre
    const double* wF;   // 3 x: weight at the I face ie+n+1, J face and K face of the ghost cell
    const double* sF;   // 3 x: wind flux through those faces
    long nw;            // entries per array
    // time series (gam_set_wind_series, apps/wind.F90 WindBC_T): n rows of
    // t, D, Vx, Vy, Vz, P, Bx, By, Bz, xBS, yBS, zBS; n = 0: the constant wind
    int n;
    double tMin, tMax, dtW, Bx0, ByC, BzC;
    const double* ts;
};

// The ionospheric inner boundary (bc[0] = 7) and its model hooks: tables
// computed on the host from the coupling fields (gam_set_ionosphere)
struct IonData {
    int on;            // the magnetosphere's hooks (HackE) run on this grid or tile
    int push, nIonP;   // PushIon on the first nIonP active shells
    double dtCpl;      // coupling time scale (code time)
    const double* Vg;  // ghost-cell velocity, 3 per (n-1) + 4 (jj + Nj kk), n = 1..4
    const double* Vp;  // PushIon's target velocity, 3 per (ii - G) + nIonP ((jj - G) + Njp (kk - G))
    const double* Ee;  // the first shell's J and K EMFs (IonEFix), 2 per jj + Nj kk
    // the wind's part (bc[1] = 4, constant wind): WindEFix and NudgeSW
    int wind;          // 1: apply them
    double vSW;        // DiffuseOuter's speed min(|vFr|, Ca)
    double dtSW0;      // NudgeSW's time scale
    const double* We;  // 7 per s + 4 (jj - G + (Njp+1) (kk - G)), s = 0..3 for i = ie-2+s: the blend
                       // weight of the I, J, K edges (negative: unchanged), their wind EMF, and
                       // DiffuseOuter's weight
    const double* Wn;  // NudgeSW's weight of the last active cell, per (jj - G) + Njp (kk - G)
};

// Ring averaging about the LFM axis (ringav.F90, gid "lfm"): rings are the k
// circles of the first NumR j rows next to each pole (GAM_BC_LFM sides),
// sliced by i (gam_set_rings)
struct RingData {
    int on, doS, doE;     // doS / doE: the pole at js / je+1 belongs to this grid
    int NumR, Np;         // rings per pole, cells per ring (Nkp)
    int recon;            // ring reconstruction: 0 PPM, 1 PLM, 2 PCM
    int nft;              // Fourier modes 0..nft removed from the fluxes (-1: none)
    int clean;            // CleanLoops
    double tScl;          // CleanLoops' scale (1 with doFastClean)
    double aScl;          // CleanRing's 2/Np (in default real)
    int Nch[32];          // chunks of ring 1..NumR
    int chunkStride;      // 5 (max chunks + 4): shared-memory chunk values of one ring
    const double* ftab;   // cos / sin (m phi_n): [(2 m + c) Np + n - 1], m = 0..2
    void* smoothE;        // smoothing EMFs, 3 components of the box (compute precision)
};

template <class R> struct DevParams {
    R gamma, gm1, CFL, pdmb, Vd0, cHogH, cHogM, dFloor, pFloor;
    R rgm1;  // 1/gm1, rounded
    int doMHD, doLFMLim, do25D, doBackground, up7;
    int doBoris;  // Boris correction with the speed of light Ca (init.F90:417-423)
    double Ca;
    int doAB3;    // third-order (AB3) predictor with ooState (init.F90:377)
    int bc[6];
    // CalcDT covers the ghost layer below / above the active range per
    // direction (1, the reference's isDT..ieDT); a tile drops it where a
    // neighbour's cells lie, the magnetosphere everywhere
    int dtKlo, dtKhi;
    int dtIlo, dtIhi, dtJlo, dtJhi;
    WindData wind;
    double inflow[8];  // uniform inner-I inflow (bc[0] = 6): rho, P, Vx, Vy, Vz, Bx, By, Bz
    IonData ion;       // ionospheric inner boundary and its hooks (bc[0] = 7)
    RingData ring;     // ring averaging about the LFM axis (bc[2] / bc[3] = 8)
};

template <class R> struct Geo {  // Grid_T arrays on the device (gamtypes.F90:168-250)
    const R* vol;    // cell
    const R* xyzcc;  // cell, 3
    const R* dl;     // cell, min(di,dj,dk)
    const R* face;   // face, 3
    const R* xfc;    // face, 9: x + 3*d
    const R* Tf;     // face, 27: n + 9*d
    const R* edge;   // edge, 3
    const R* Te;     // edge, 27: n + 9*d
    const R* Teb;    // edge, 12: q + 4*d
    // FP32 form only: face centroid minus cell centroid for the six faces of
    // a cell, x + 3*f with f = I-, I+, J-, J+, K-, K+ (computed in FP64, rounded
    // once). Replaces xfc and xyzcc in bFlux2Fld, whose absolute coordinates
    // lose the cell-size differences when rounded to FP32.
    const R* dxf;    // cell, 18
    // geometry-only operands of the reconstructions, made with the geometry
    // (gam_geom_tables; null in the differentiation form): the 8CENT interpolant
    // of the volumes at the faces of each direction and its reciprocal. The
    // forms that multiply by the reciprocal keep only that one.
    const R* vif;    // face, 3
    const R* rvif;   // face, 3
    // the same of the areas at the edges (dT1 faces along dT2, then dT2 faces
    // along dT1, per edge direction), and 1/(determinant of the edge's B map)
    const R* fae;    // edge, 6: q + 2*eD
    const R* rfae;   // edge, 6
    const R* rdet;   // edge, 3
    const double* fcB0;    // face, 9  (background; FP64 in both forms)
    const double* bFlux0;  // face, 3
    const double* edgB0;   // edge, 6: c + 2*d
    const double* B0;      // cell, 3
    const double* dpB0;    // cell, 3
};

template <class R> struct StateBuf {
    R* Gas;  // cell, 5
    R* mf;   // face, 3
    R* B;    // cell, 3
};

template <class R> struct Work {
    R* QW;   // cell, 5: volume * primitives of the half state (BlockCon2Prim), the recon operand
    R* QB;   // cell, 3: volume * Bxyz of the half state
    R* Dh;   // cell, 1: half-state density (GetCornerD)
    R* Wn;   // cell, 5: limiter primitives (state n with lfmlim, else the half state)
    R* Bl;   // cell, 3: limiter Bxyz without lfmlim (= half-state Bxyz); lfmlim uses State%Bxyz
    R* VdV;  // cell, 3: volume * momentum / max(density, dFloor) of the half state
    R* abh;  // face, 3: area * (half-state flux / max(area, TINY)), the EdgeLRs recon operand
    R* bn;   // face, 3: limiter flux / max(area, TINY)
    R* Bnf;  // face, 3: half-state flux / area
    R* AVf;  // cell, 9: area(dT1) * Vf(x) for edge direction eD at x + 3*eD
    R* E;    // edge, 3
    R* gF;   // face, 15: gas flux v + 5*d (already times face area)
    R* mF;   // face, 9: magnetic flux x + 3*d
    // differentiation form only (null in the step): the flux kernels' face
    // states, 22 per face and direction, q + 22*d: WL, WR (5 each), MagL,
    // MagR (3 each), VaD and the diffusion sums dW (5)
    R* fsv;
    // differentiation form only: the edge kernels' corner values, 10 per
    // edge and direction, q + 10*eD: Dc, bT1L, bT1R, fA1, bT2L, bT2R, fA2, VC (3)
    R* esv;
};
constexpr int GAM_FSV_NC = 22;
constexpr int GAM_ESV_NC = 10;

struct Range {  // inclusive box-index range
    int i0, i1, j0, j1, k0, k1;
};


// The tile of one block of the flux kernel of direction D, and its stencil
// boxes in shared memory: TX faces in i by TN along j (D = 0, 1) or k (D = 2);
// reconstruction operands of cells -4..3 and limiter values of cells -2..1
// along D. On the I sweep both boxes start 4 cells below the tile's first face
// (a TMA box starts on a 16-byte boundary: an even cell in FP64, a multiple of
// 4 in FP32; the flux ranges start at cell 4 and tiles are 16 or 32 wide). The I
// sweep's boxes are 8 cells wider than its tile; 16 x 8 faces instead of 32 x 4
// fit a grid's odd extents better: 192^3 strict 858 -> 782 us, FP32 296 -> 280,
// 96^3 125 -> 113 and 47 -> 43.
template <class R, int D> struct FluxTile {
    static constexpr int TX = D == 0 || sizeof(R) == 8 ? 16 : 32;
    static constexpr int TN = 8;
    static constexpr int NT = TX * TN;
    static constexpr int QX = D == 0 ? TX + 8 : TX;
    static constexpr int QN = D == 0 ? TN : TN + 7, LN = D == 0 ? TN : TN + 3;
    static constexpr unsigned BYTES = 8u * (QN + LN) * QX * sizeof(R), BYTES_GAS = 5u * (QN + LN) * QX * sizeof(R);
    static constexpr unsigned LOFF = 8u * QN * QX * sizeof(R), SMEM = BYTES;
    static_assert(5 * QN * QX * sizeof(R) % 128 == 0 && LOFF % 128 == 0 && 5 * LN * QX * sizeof(R) % 128 == 0,
                  "TMA destinations are 128-byte aligned");
};
// The tensor maps of those boxes for one direction: the reconstruction
// operands, the limiter primitives and the limiter field
struct GamFluxMaps {
    CUtensorMap QW, QB, Wn, Bl;
};
// The tile of one block of the edge-EMF kernel of direction E (dT1 = E+1, dT2 =
// E+2) and its boxes in shared memory, one after the other: 0, 1 the EdgeLRs
// operands of dT1 faces along dT2 and of dT2 faces along dT1 (cells -4..3), 2
// the three components of GetCornerV's operand (along dT2), 3, 4 the limiter
// values of 0, 1 (-2..1), 5 the density (-1..0 along both). A box that extends
// along i starts 4 below the tile (16-byte boundary, see FluxTile).
template <int E> struct EdgeTile {
    static constexpr int d1 = (E + 1) % 3, d2 = (E + 2) % 3;
    static constexpr int T0 = E == 0 ? 16 : 32, T1 = E == 0 ? 4 : (E == 1 ? 1 : 8), T2 = E == 0 ? 4 : (E == 1 ? 8 : 1);
    static constexpr int NT = T0 * T1 * T2;
    __host__ __device__ static constexpr int T(int d) { return d == 0 ? T0 : d == 1 ? T1 : T2; }
    __host__ __device__ static constexpr bool along(int q, int d) {
        return (q == 0 || q == 2 || q == 3) ? d == d2 : (q == 1 || q == 4) ? d == d1 : d != E;
    }
    __host__ __device__ static constexpr int org(int q, int d) {
        return !along(q, d) ? 0 : d == 0 ? 4 : q < 3 ? 4 : q < 5 ? 2 : 1;
    }
    __host__ __device__ static constexpr int ext(int q, int d) {
        return T(d) + (!along(q, d) ? 0 : d == 0 ? 8 : q < 3 ? 7 : q < 5 ? 3 : 1);
    }
    __host__ __device__ static constexpr int size(int q) { return ext(q, 0) * ext(q, 1) * ext(q, 2); }
    __host__ __device__ static constexpr int off(int q) {
        int o = 0;
        for (int p = 0; p < q; p++) o += size(p) * (p == 2 ? 3 : 1);
        return o;
    }
    __host__ __device__ static constexpr int str(int q, int d) {
        return d == 0 ? 1 : d == 1 ? ext(q, 0) : ext(q, 0) * ext(q, 1);
    }
    // position of the tile's point (x, y, z) in box q
    __host__ __device__ static constexpr int at(int q, int x, int y, int z) {
        return off(q) + ((z + org(q, 2)) * ext(q, 1) + y + org(q, 1)) * ext(q, 0) + x + org(q, 0);
    }
    __host__ __device__ static constexpr int all() { return off(6); }
};
struct GamEdgeMaps {
    CUtensorMap m[6];
};
struct GamFluxMapSet {
    GamFluxMaps m[2][3];  // [State buffer][direction]
    GamEdgeMaps e[3];     // [edge direction]
};

// Everything one step launch needs.
template <class R> struct Ctx {
    GamBox b;
    DevParams<R> P;
    Geo<R> g;
    StateBuf<R> st[2];   // double buffer: st[cur] = State (n), st[1-cur] = oState (n-1) -> State (n+1)
    R* oomf;             // doAB3: ooState face fluxes (n-2), refreshed from oState by k_update_faces
    Work<R> w;
    GamScalars* sc;
    const GamFluxMapSet* fmaps;  // host memory, with the handle
    double gamma, gm1;
    // side streams and fork/join events of the step graph (independent
    // kernels of a step run as parallel branches); null: one stream
    cudaStream_t aux[5];
    cudaEvent_t ev[8];
};
