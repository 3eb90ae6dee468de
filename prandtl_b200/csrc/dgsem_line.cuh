// dgsem_line.cuh -- FP64 right-hand side by lines (sm_100a): Euler and
// Navier-Stokes with contravariant viscous fluxes on affine elements.
//
// One lane owns one line of its element per direction: it loads the line's
// primitives from shared memory into registers, evaluates the line's
// Np(Np-1)/2 two-point fluxes and its two face fluxes, and keeps the line's
// Np x NF sums in registers; the directions hand their sums on through one
// [NF][nodes] buffer in shared memory, and the lines of the last direction end
// with the nodes' right-hand sides in registers and write the epilogue.
//
// The general form (dgsem_impl.cuh) evaluates pairs into shared memory and sums
// them per node.  It was bound by shared-memory wavefronts (70 % of peak at 3D
// Np = 4), instruction count and instruction-cache misses at 16 warps per SM.
// Here a node's primitives are read once per direction instead of once per
// pair, no two-point or face flux goes through shared memory, every lane has
// work in every phase and boundary and blending code is compiled in only where
// it is used: half the warp instructions (157 M -> 73 M at 32^3 Np = 4).  What
// bounds it now is FP64 issue (53 % of the pipe) and the latency of the global
// loads at 12 warps per SM.  Measured, one launch:
//   3D Np = 4 Navier-Stokes, 32^3 elements   324 -> 147 us
//   3D Np = 5 Navier-Stokes, 15^3            103 ->  49 us
//   3D Np = 4 Euler, 24^3                    114 ->  52 us
//   2D Np = 4 Euler, blended, 256^2          107 ->  57 us
//   2D Np = 5 Euler, 101^2                    35 ->  23 us
#pragma once

namespace prandtl {
namespace {

// Lane and shared-memory layout.  NL lanes (the lines of one direction) own
// one element.  Elements are packed into warps where that fills at least 30
// of the 32 lanes (the group then synchronises with __syncwarp), else into
// the CTA's threads (__syncthreads).  A field row holds node (x, y, z) at
// x + SY y + SZ z; SY, SZ and the elements' stride keep the 16
// lanes of an 8-byte access on distinct banks for the lines of every direction
// (found by enumeration: 3D Np = 4 takes 2.7 wavefronts per access against 6
// without padding).
template <int DIM, int NP, typename W = double>
struct LineShape {
    static constexpr bool F64 = sizeof(W) == 8;
    static constexpr int ND = ipow(NP, DIM), NL = ND / NP, NF = DIM + 2;
    static constexpr int SY = DIM == 2 ? (F64 || NP % 2 == 0 ? NP + 1 : NP) : NP;
    static constexpr int SZ = DIM == 2 ? 0 : (NP == 2 ? 5 : NP == 3 ? 9 : NP == 4 ? (F64 ? 19 : 16) : NP == 5 ? 25 : (F64 ? 39 : 36));
    static constexpr int ROW = (NP - 1) * (1 + SY + SZ) + 1;
    // element stride, modulo the 16 double / 32 float banks, that spreads a
    // half-warp's / warp's elements over the banks
    static constexpr int BANKS = F64 ? 16 : 32, BYTES = sizeof(W);
    static constexpr int STRIDE = F64 ? (DIM == 2 ? (NP == 2 ? 2 : NP == 3 ? 3 : NP == 4 ? 4 : NP == 5 ? 5 : 10)
                                                  : (NP == 2 ? 12 : NP == 3 ? 11 : NP == 4 ? 12 : NP == 5 ? 13 : 4))
                                      : (DIM == 2 ? (NP == 2 ? 10 : NP == 3 ? 9 : NP == 4 ? 28 : NP == 5 ? 8 : 10)
                                                  : (NP == 2 ? 12 : NP == 3 ? 27 : NP == 4 ? 5 : NP == 5 ? 25 : 9));
    static constexpr int padded(int end) { return end + (STRIDE + BANKS - end % BANKS) % BANKS; }
    static constexpr int EPW = NL <= 32 ? 32 / NL : 0;
    static constexpr bool WARP = EPW * NL >= 30;
    // threads per CTA when elements are packed into the CTA: 125 of 128 lanes at
    // 3D Np = 5, 126 at Np = 3, 252 of 256 at Np = 6
    static constexpr int THREADS = (!WARP && NL > 32) ? 256 : 128;
    static constexpr int EPB = WARP ? (THREADS / 32) * EPW : THREADS / NL;
    static_assert(EPB >= 1 && EPB * NL <= THREADS && THREADS % 32 == 0 && EPW * NL <= 32, "lanes of a CTA and of a warp");
};
constexpr size_t MAX_SMEM = 227 * 1024;   // shared memory a CTA can have
// The right-hand side's shared area of an element.
template <int DIM, int NP>
struct RhsLineShape : LineShape<DIM, NP> {
    using L = LineShape<DIM, NP>;
    // field rows: rho, v, beta (the two-point fluxes), then 1/beta and |v| + c (surface fluxes)
    static constexpr int RHO = 0, V = 1, BETA = 1 + DIM, RBETA = 2 + DIM, LAM = 3 + DIM, K = 4 + DIM;
    static constexpr int NQ = 2 + DIM;                  // rows the two-point fluxes read
    // then the directions' running sums, and the element's constants: the neighbour
    // table (2 DIM entries of two int2), the faces' normals and their lengths,
    // adj(J) and det J
    static constexpr int NBR = (K + L::NF) * L::ROW, NOR = NBR + 4 * DIM, GEO = NOR + 2 * DIM * (DIM + 1);
    static constexpr int PER_ELEM = L::padded(GEO + DIM * DIM + 1);
    static_assert(GEO + DIM * DIM + 1 <= PER_ELEM && 3 * L::NL <= L::NF * L::ROW, "an element's shared area");
    static_assert(sizeof(double) * L::EPB * PER_ELEM + CTX_RESERVE <= MAX_SMEM, "a CTA's shared memory");
};

// Resident CTAs the register budget is sized for: 168 registers a thread.  A
// line's sums and primitives take 80 (3D, Np = 4); at 128 registers the 3D
// kernels spill in the two-point fluxes (32^3 Np = 4 Navier-Stokes 157 -> 228 us,
// 24^3 Euler 52 -> 60 us), and more than 168 gives up resident warps (2D Np = 5
// Euler 22.9 -> 25.4 us, 3D Np = 5 Euler 69 -> 81 us at 255).  The 3D Np = 5
// Navier-Stokes kernel alone, whose viscous rows come on top, is faster with 255
// (20^3: 123 -> 97 us).  The batch's other two launch shapes (V = 1, 2) have 255
// and 128.
template <int DIM, int NP, bool NS, int V = 0>
constexpr int line_min_blocks() {
    return cmax(1, 65536 / ((V == 1 || (V == 0 && NS && DIM == 3 && NP == 5) ? 255 : V == 2 ? 128 : 168) *
                            LineShape<DIM, NP>::THREADS));
}

// The FP32-bulk kernels: 96 registers up to Np = 4, 128 beyond (ensemble N=2 and
// N=4 lifts 48 and 284 us at 96, 51 and 230 us at 128; 80 is slower everywhere).
template <int DIM, int NP, typename W>
constexpr int lift_line_min_blocks() {
    return sizeof(W) == 8 ? line_min_blocks<DIM, NP, false>()
                          : cmax(1, 65536 / ((NP <= 4 ? 96 : 128) * LineShape<DIM, NP, W>::THREADS));
}

// Logarithmic mean of x, y > 0 in the form q = (x+y) / (2 mean), with
// f = (y-x)/(y+x) and u = f^2: q = atanh(f)/f = 1 + u/3 + u^2/5 + ...
// (ComputeLogMean, BasicOperations.cpp:6-12).  Near means (u < 1e-4, the
// reference's own series branch): four terms, truncation below 2e-17.
__device__ __forceinline__ double log_q_near(double u) {
    return u * (1.0 / 3.0 + u * (1.0 / 5.0 + u * (1.0 / 7.0)));   // q - 1
}
// Further apart: the series to u^11 up to u = 0.04 (ratios up to 3/2,
// truncation below 2e-18), which loses no digits to the logarithm of a ratio
// near one; beyond that the logarithm.  Not inlined: seldom taken, and its code
// would push the hot path out of the instruction cache.
__device__ __noinline__ double log_q_far(double x, double y, double f, double u) {
    if (u < 0.04) {
        double p = 1.0 / 23.0;
#pragma unroll
        for (int k = 21; k >= 1; k -= 2) p = fma(p, u, 1.0 / k);
        return p;
    }
    return 0.5 * log(y / x) / f;
}

// sqrt(x): hardware estimate of 1/sqrt (PTX rsqrt.approx.ftz.f64) refined by a
// coupled (Goldschmidt) iteration (Markstein, IBM J. Res. Dev. 34 (1990)
// 111-119).  Outside the positive normal numbers, which one integer compare of
// the high word tells, as sqrt has it: NaN for negative arguments (a state
// without a speed of sound must not look like one), zero, infinity and NaN
// themselves; subnormals too come back as they are, within 2e-154 of their root.
__device__ __forceinline__ double sqrt_pos(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double g = x * r, h = 0.5 * r;
    const double e = fma(-g, h, 0.5);
    g = fma(g, e, g);
    h = fma(h, e, h);
    const double d = fma(-g, g, x);
    g = fma(d, h, g);
    if ((unsigned)__double2hiint(x) - 0x00100000u >= 0x7fe00000u) g = x < 0.0 ? nan("") : x;
    return g;
}

// A load that stays where it is written: the compiler may not sink it to its
// first use behind the arithmetic meant to hide its latency.
__device__ __forceinline__ double ldg_now(const double *p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Brings the lines that hold p[0..n) into L2, spread over the NL lanes of an
// element, without a register or a wait: for operands read later from DRAM.
__device__ __forceinline__ void prefetch_l2(const double *p, int n, int ln, int nl) {
    for (int q = 16 * ln; q < n; q += 16 * nl) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + q));
}

// Two-point flux along the metric row m (ChandrashekarFlux.cpp:11-83) of nodes
// (rho, v, beta), rearranged: with q = (x+y)/(2 mean) of rho and beta and
// rs = 1/(beta_a + beta_b), the enthalpy term p_hat/rho_ln + 1/(2(g-1) beta_ln)
// is rs (q_rho + q_beta/(g-1)), and |v_mean|^2 - (|v_a|^2 + |v_b|^2)/4 is
// v_a.v_b/2.  NEAR: the caller has checked that both means are near.
template <int DIM, bool NEAR>
__device__ __forceinline__ void line_flux(const double *a, const double *b, const double *m, double gm1i, double *F) {
    const double sr = a[0] + b[0], sb = a[1 + DIM] + b[1 + DIM];
    const double rr = rcp(sr), rs = rcp(sb);
    const double fr = (b[0] - a[0]) * rr, fb = (b[1 + DIM] - a[1 + DIM]) * rs;
    const double ur = fr * fr, ub = fb * fb;
    double qr, qb, rho_ln4;   // rho_ln4: rho_ln / 2 (the sum of velocities stands for twice their mean)
    if constexpr (NEAR) {
        const double ar = log_q_near(ur);
        qr = 1.0 + ar;
        qb = 1.0 + log_q_near(ub);
        rho_ln4 = (0.25 * sr) * fma(-ar, fma(-ar, 1.0 - ar, 1.0), 1.0);
    } else {
        qr = log_q_far(a[0], b[0], fr, ur);
        qb = log_q_far(a[1 + DIM], b[1 + DIM], fb, ub);
        rho_ln4 = (0.25 * sr) * rcp(qr);
    }
    double vs[DIM], vn = 0.0, dot = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        vs[d] = a[1 + d] + b[1 + d];
        vn = fma(vs[d], m[d], vn);
        dot = fma(a[1 + d], b[1 + d], dot);
    }
    const double p_hat = (0.5 * sr) * rs;
    const double h = fma(0.5, dot, rs * fma(gm1i, qb, qr));
    F[0] = rho_ln4 * vn;
    const double hF = 0.5 * F[0];
#pragma unroll
    for (int d = 0; d < DIM; ++d) F[1 + d] = fma(hF, vs[d], p_hat * m[d]);
    F[1 + DIM] = F[0] * h;
}

// Primitive variables of a trace: (rho, v, beta, 1/beta, |v| + c).
template <int DIM>
__device__ __forceinline__ void line_prim(const double *s, double gamma, double gammaM1, double *q) {
    constexpr int NF = DIM + 2;
    const double r = rcp(s[0]);
    double vsq = 0.0;
    q[0] = s[0];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        q[1 + d] = s[1 + d] * r;
        vsq = fma(q[1 + d], q[1 + d], vsq);
    }
    const double p = gammaM1 * fma(-0.5 * s[0], vsq, s[NF - 1]);
    q[1 + DIM] = 0.5 * s[0] * rcp(p);
    const double pr = p * r;
    q[2 + DIM] = 2.0 * pr;
    q[3 + DIM] = sqrt_pos(vsq) + sqrt_pos(gamma * pr);
}

// Surface flux of traces a, b along nor (ChandrashekarFlux.cpp:85-161), the
// two-point flux in line_flux's arrangement minus the dissipation.  nlen = |nor|.  quirk3:
// the reference's 3D energy dissipation (:131).
template <int DIM>
__device__ __forceinline__ void line_face_flux(const double *a, const double *b, const double *nor, double nlen,
                                               double gm1i, bool quirk3, bool dissipation, double *F) {
    constexpr int NF = DIM + 2;
    const double sr = a[0] + b[0], sb = a[1 + DIM] + b[1 + DIM];
    const double dr = b[0] - a[0];
    const double rr = rcp(sr), rs = rcp(sb);
    const double fr = dr * rr, fb = (b[1 + DIM] - a[1 + DIM]) * rs;
    const double ur = fr * fr, ub = fb * fb;
    double qr = 1.0 + log_q_near(ur), qb = 1.0 + log_q_near(ub);
    if (!(ur < 1e-4)) qr = log_q_far(a[0], b[0], fr, ur);
    if (!(ub < 1e-4)) qb = log_q_far(a[1 + DIM], b[1 + DIM], fb, ub);
    const double rm = 0.5 * sr;
    double vs[DIM], vn = 0.0, dot = 0.0, dvv = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        vs[d] = a[1 + d] + b[1 + d];
        const double dv = b[1 + d] - a[1 + d];
        vn = fma(vs[d], nor[d], vn);
        dot = fma(a[1 + d], b[1 + d], dot);
        if (DIM == 3 && d == 2 && quirk3) dvv += dv + 0.5 * vs[d] * rcp(rm);   // rho_mean dv + v_mean
        else dvv = fma(0.5 * dv, vs[d], dvv);
    }
    const double p_hat = rm * rs;
    const double h = fma(0.5, dot, rs * fma(gm1i, qb, qr));
    // 1/beta_ln = 2 rs q_beta
    const double diss = 0.5 * dr * fma(2.0 * gm1i, rs * qb, dot) +
                        rm * fma(0.5 * gm1i, b[2 + DIM] - a[2 + DIM], dvv);
    const double hl = dissipation ? 0.5 * dmax(a[3 + DIM], b[3 + DIM]) * nlen : 0.0;
    const double F0 = (0.5 * rm) * rcp(qr) * vn, hF = 0.5 * F0;
    F[0] = fma(-hl, dr, F0);
#pragma unroll
    for (int d = 0; d < DIM; ++d)
        F[1 + d] = fma(-hl, b[0] * b[1 + d] - a[0] * a[1 + d], fma(hF, vs[d], p_hat * nor[d]));
    F[NF - 1] = fma(F0, h, -hl * diss);
}

// Node strides of direction `dir`: line ln has its first node at
// sa (ln % NP) + sb (ln / NP) and its nodes st apart.
template <int DIM>
__device__ __forceinline__ void line_strides(int dir, int sy, int sz, int &sa, int &sb, int &st) {
    sa = dir == 0 ? sy : 1;
    sb = DIM == 2 ? 0 : (dir == 2 ? sy : sz);
    st = dir == 0 ? 1 : (dir == 1 ? sy : sz);
}

// The RHS values al of NP nodes (node0 + i * step) to the call's result: dudt,
// or the fused Runge-Kutta stage update with the state check of the new state
// (non-finite values, rho <= 0, p <= 0; one atomic per violating node).  The
// global operands of two nodes are in flight together.
template <int NP, int NF>
__device__ __forceinline__ void rk_epilogue(const ElemIO &a, const double (*al)[NF], long long node0, int step) {
    const long long Ndof = a.Ndof;
    const int mode = a.mode;
    if (mode == EPI_STORE) {
#pragma unroll
        for (int i = 0; i < NP; ++i)
#pragma unroll
            for (int f = 0; f < NF; ++f) a.dudt[f * Ndof + node0 + i * step] = al[i][f];
        return;
    }
    const bool need_b = (mode == EPI_LSRK && a.rkA != 0.0) || mode == EPI_SSP2 || mode == EPI_SSP3;
    const double *pb = mode == EPI_LSRK ? a.du : a.x0;
    const double cx = mode == EPI_SSP2 ? 3. / 4 : 1. / 3, cy = mode == EPI_SSP2 ? 1. / 4 : 2. / 3;
    constexpr int KB = 6 * NP * NF <= 128 ? NP : (NP + 1) / 2;
#pragma unroll
    for (int i0 = 0; i0 < NP; i0 += KB) {
        double ua[KB][NF], ub[KB][NF];
#pragma unroll
        for (int k = 0; k < KB; ++k)
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const long long g = f * Ndof + node0 + (i0 + k) * step;
                ua[k][f] = i0 + k < NP ? __ldg(a.u + g) : 0.0;
                ub[k][f] = i0 + k < NP && need_b ? pb[g] : 0.0;
            }
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            if (i0 + k >= NP) continue;
            const long long gnode = node0 + (i0 + k) * step;
            double v[NF];
            bool finite = true;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const double L = al[i0 + k][f];
                if (mode == EPI_LSRK) {
                    const double dv = need_b ? a.rkA * ub[k][f] + a.dt * L : a.dt * L;
                    a.du[f * Ndof + gnode] = dv;
                    v[f] = ua[k][f] + a.rkB * dv;
                } else {
                    const double y = ua[k][f] + a.dt * L;
                    v[f] = mode == EPI_SSP1 ? y : cx * ub[k][f] + cy * y;
                }
                a.u_out[f * Ndof + gnode] = v[f];
                finite = finite && isfinite(v[f]);
            }
            if (a.health) {
                unsigned bad = finite ? 0u : 1u;
                if (finite) {
                    double mm = 0.0;
#pragma unroll
                    for (int f = 1; f < NF - 1; ++f) mm += v[f] * v[f];
                    if (!(v[0] > 0.0)) bad |= 2u;
                    else if (!(2.0 * v[0] * v[NF - 1] - mm > 0.0)) bad |= 4u;
                }
                if (bad) atomicOr(a.health, bad);
            }
        }
    }
}

// What the end node's RHS receives (times w0 J) from a boundary face of local
// side `side`, inner trace s0, own viscous row v0: the viscous flux of the
// accepted types minus the boundary flux along the outward normal
// (BdrFaceIntegrator.cpp:61-186).  Not inlined: few faces are boundary faces,
// and its code (powers, every condition) is long.
template <int DIM, bool NS>
__device__ __noinline__ void line_boundary_flux(const BcDev &bc, const PhysParams &P, int side, const double *io,
                                                double *face) {
    constexpr int NF = DIM + 2;
    const double *s = io, *nor = io + NF, *v0 = io + NF + DIM;
    double fb[NF], fv[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) fv[f] = 0.0;
    boundary_flux<DIM, double>(bc, s, nor, P, 0.0, fb);
    if constexpr (NS) {
        // Fv(inner state, inner gradients) . n for the no-slip walls and supersonic
        // outflow; the other accepted types evaluate Fv with zero gradients
        if (bc.type == BC_NOSLIP_ADIABATIC || bc.type == BC_NOSLIP_ISOTHERMAL || bc.type == BC_OUTFLOW) {
            const double so = side ? 1.0 : -1.0;
#pragma unroll
            for (int f = 1; f < NF; ++f) fv[f] = so * v0[f - 1];
            if (bc.type == BC_NOSLIP_ADIABATIC) {   // NoSlipAdiabWallBdrFaceIntegrator.cpp:17-31
                double nn = 0.0, w = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    nn += nor[d] * nor[d];
                    w += bc.wall_vel[d] * fv[1 + d];
                }
                fv[NF - 1] = w + bc.heat_flux * sqrt(nn);
            }
        }
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) face[f] = fv[f] - fb[f];
}
// ... its operands copied, so that the caller's arrays stay in registers
template <int DIM, bool NS>
__device__ __forceinline__ void line_boundary(const ElemIO &a, const PhysParams &P, int cond, const double *nor,
                                              const double *s0, const double *v0, int side, double *face) {
    constexpr int NF = DIM + 2;
    double in[2 * NF + DIM - 1], out[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) in[f] = s0[f];
#pragma unroll
    for (int d = 0; d < DIM; ++d) in[NF + d] = nor[d];
#pragma unroll
    for (int f = 0; f < NF - 1; ++f) in[NF + DIM + f] = v0[f];
    line_boundary_flux<DIM, NS>(a.bcs[cond], P, side, in, out);
#pragma unroll
    for (int f = 0; f < NF; ++f) face[f] = out[f];
}

// One element of a lane group: lane `ln` of NL, `sH` the element's shared area.
// Every thread of the synchronising group calls it; lanes without an element
// or a line have ok = false.  SYNC orders the group's shared memory.
// REF: Navier-Stokes in the reference mode (quirks == 0), whose viscous rows
// come in two parts: the volume's, of the element's last node's state
// (DGSEMIntegrator.cpp:620), and the face nodes' own (lift_line_element).  The
// general form reads 15 gradients per node, twice per face node, and evaluates
// viscous fluxes from them at 12 warps per SM; here 18 values per node pass
// through memory.  20^3 Np = 4: RHS 145 -> 57 us, lifting 49 -> 40 us.
template <int DIM, int NP, bool NS, bool BLEND, bool BC, bool REF, typename Sync>
__device__ __forceinline__ void rhs_line_element(const ElemIO &a, const PhysParams &P, const OpTables &T, int e, bool ok,
                                                 double *sH, int ln, const Sync &sync) {
    using L = RhsLineShape<DIM, NP>;
    constexpr int ND = L::ND, NL = L::NL, NF = L::NF, ROW = L::ROW, NQ = L::NQ;
    double *sA = sH + L::K * ROW;   // the directions' running sums [NF][ROW]
    const long long Ndof = a.Ndof, e0 = (long long)e * ND;
    const double gamma = P.gamma, gm1 = P.gammaM1, gm1i = P.gammaM1Inverse;
    const bool quirk3 = REF || (!NS && P.quirks == 0);
    static_assert(!REF || (NS && !BLEND && !BC), "the reference mode's lines are for plain Navier-Stokes solves");
    const double *gface = reinterpret_cast<const double *>(a.grad) + Ndof * (DIM * (NF - 1));   // REF: [E][2 DIM][NF-1][NL]
    // a lane's nodes in the node-wise phases: ln, ln + NL, ... (those of its last-direction line)
    const int own0 = ln % NP + L::SY * (DIM == 2 ? 0 : ln / NP);
    constexpr int own_st = DIM == 2 ? L::SY : L::SZ;

    // ---- primitives of the lane's nodes; largest |v| + c
    double lam = 0.0;
    int2 *sNbr = reinterpret_cast<int2 *>(sH + L::NBR);   // {element, local face}, {face, role}
    double *sNor = sH + L::NOR, *sGeo = sH + L::GEO;
    if (ok) {
        // the element's tables: loads issued with the state's, the normals (which
        // wait for the table) stored after the primitives' arithmetic
        constexpr int NG = (DIM * DIM + NL) / NL, NB = (2 * DIM + NL - 1) / NL;
        int4 nb[NB];
        double g[NG], nor[NB][DIM], s[NP][NF];
#pragma unroll
        for (int k = 0; k < NB; ++k)
            nb[k] = __ldg(a.nbr + (long long)e * (2 * DIM) + min(ln + k * NL, 2 * DIM - 1));
#pragma unroll
        for (int i = 0; i < NP; ++i)
#pragma unroll
            for (int f = 0; f < NF; ++f) s[i][f] = ldg_now(a.u + f * Ndof + e0 + ln + NL * i);
#pragma unroll
        for (int k = 0; k < NG; ++k) g[k] = __ldg(a.geo + (long long)e * (DIM * DIM + 1) + min(ln + k * NL, DIM * DIM));
        // what is read after the two-point fluxes: the element's viscous rows (32^3
        // Np = 4: 157 -> 148 us) and, of states that leave L2 between stages (above
        // 3 M values, 24 MB: the stage touches three to four times that), the stage
        // update's other operand (256^2 step 160 -> 156 us; smaller states, 1 % slower)
        if constexpr (NS) prefetch_l2(reinterpret_cast<const double *>(a.grad) + e0 * (DIM * (NF - 1)), DIM * (NF - 1) * ND, ln, NL);
        if (NF * Ndof > 3000000 && (a.mode == EPI_LSRK ? a.rkA != 0.0 : a.mode >= EPI_SSP2))
#pragma unroll
            for (int f = 0; f < NF; ++f) prefetch_l2((a.mode == EPI_LSRK ? a.du : a.x0) + f * Ndof + e0, ND, ln, NL);
#pragma unroll
        for (int k = 0; k < NB; ++k)
#pragma unroll
            for (int d = 0; d < DIM; ++d) nor[k][d] = ldg_now(a.fnor + (long long)nb[k].z * DIM + d);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            double q[L::K];
            line_prim<DIM>(s[i], gamma, gm1, q);
#pragma unroll
            for (int k = 0; k < L::K; ++k) sH[k * ROW + own0 + i * own_st] = q[k];
            lam = fmax(lam, q[L::LAM]);
        }
#pragma unroll
        for (int k = 0; k < NG; ++k)
            if (ln + k * NL < DIM * DIM + 1) sGeo[ln + k * NL] = g[k];
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            const int lf = ln + k * NL;
            if (lf < 2 * DIM) {
                sNbr[2 * lf] = make_int2(nb[k].x, nb[k].y);
                sNbr[2 * lf + 1] = make_int2(nb[k].z, nb[k].w);
                double nn = 0.0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    sNor[lf * (DIM + 1) + d] = nor[k][d];
                    nn = fma(nor[k][d], nor[k][d], nn);
                }
                sNor[lf * (DIM + 1) + DIM] = sqrt_pos(nn);
            }
        }
    }
    if (a.lambda) {
        for (int o = 16; o > 0; o >>= 1) lam = fmax(lam, __shfl_xor_sync(0xffffffffu, lam, o));
        if ((threadIdx.x & 31) == 0) atomic_max_seen(a.lambda, lam);
    }
    sync();

    // ---- blending coefficient (PerssonPeraireIndicator.cpp:21-58, DGSEMOperator.cpp:60-80)
    double alpha = 0.0;
    if (BLEND && P.blending) {
        double *b0 = sA, *b1 = sA + ROW;
        if (ok) {
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                const int n = own0 + i * own_st;
                const double rho = sH[n];
                b0[n] = rho * (0.5 * sH[L::RBETA * ROW + n] * rho);   // rho p
            }
        }
        sync();
        double md[NP];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {   // modes along each line, last direction left in registers
            const double *in = (d & 1) ? b1 : b0;
            double *out = (d & 1) ? b0 : b1;
            int sa, sb, st;
            line_strides<DIM>(d, L::SY, L::SZ, sa, sb, st);
            const int n0 = sa * (ln % NP) + sb * (ln / NP);
            if (ok) {
                double x[NP];
#pragma unroll
                for (int l = 0; l < NP; ++l) x[l] = in[n0 + l * st];
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    md[i] = 0.0;
#pragma unroll
                    for (int l = 0; l < NP; ++l) md[i] = fma(T.Vinv[i * NP + l], x[l], md[i]);
                    if (d < DIM - 1) out[n0 + i * st] = md[i];
                }
            }
            sync();
        }
        // the lines' modal energies: all modes, without the highest, without the two highest
        if (ok) {
            const int mx = max(ln % NP, DIM == 2 ? 0 : ln / NP);
            double en[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                const double m2 = md[i] * md[i];
                en[0] += m2;
                if (i <= NP - 2 && mx <= NP - 2) en[1] += m2;
                if (i <= NP - 3 && mx <= NP - 3) en[2] += m2;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) sA[k * NL + ln] = en[k];   // 3 NL <= NF ROW
        }
        sync();
        if (ok) {
            double s0 = 0.0, s1 = 0.0, s2 = 0.0;
            for (int q = 0; q < NL; ++q) {   // every lane in the same order
                s0 += sA[q];
                s1 += sA[NL + q];
                s2 += sA[2 * NL + q];
            }
            double eta = 1.0 - s1 / s0;
            eta = fmax(eta, 1.0 - s2 / s1);
            const double thr = P.modal_threshold;
            double al = 1.0 / (1.0 + exp(-9.21024 * (eta - thr) / thr));
            if (al < P.alpha_min) al = 0.0;
            else if (al > 1.0 - P.alpha_min) al = 1.0;
            alpha = fmin(al, P.alpha_max);
            if (ln == 0 && a.alpha) a.alpha[e] = alpha;
        }
        sync();   // the sums' buffer is read no more
    }

    // ---- per direction: volume, subcell and surface terms of the lane's line
    const double *grad = reinterpret_cast<const double *>(a.grad);
    const double rw0 = 1.0 / T.w[0];
    double al[NP][NF];
#pragma unroll 1
    for (int dir = 0; dir < DIM; ++dir) {
        int sa, sb, st;
        line_strides<DIM>(dir, L::SY, L::SZ, sa, sb, st);
        const int n0 = sa * (ln % NP) + sb * (ln / NP);
        double q[NP][NQ], m[DIM];
        bool far = false;
#pragma unroll
        for (int i = 0; i < NP; ++i)
#pragma unroll
            for (int k = 0; k < NQ; ++k) q[i][k] = 1.0;
        if (ok) {
#pragma unroll
            for (int i = 0; i < NP; ++i)
#pragma unroll
                for (int k = 0; k < NQ; ++k) q[i][k] = sH[k * ROW + n0 + i * st];
#pragma unroll
            for (int d = 0; d < DIM; ++d) m[d] = sGeo[dir * DIM + d];
            // all of the line's means near: u of any two nodes is at most that of
            // the smallest and the largest value
            double lo[2] = {q[0][0], q[0][1 + DIM]}, hi[2] = {q[0][0], q[0][1 + DIM]};
#pragma unroll
            for (int i = 1; i < NP; ++i)
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const double v = q[i][k * (1 + DIM)];
                    lo[k] = v < lo[k] ? v : lo[k];
                    hi[k] = v > hi[k] ? v : hi[k];
                }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const double d = hi[k] - lo[k], s = hi[k] + lo[k];
                far = far || !(d * d < 1e-4 * (s * s));
            }
        }
        // the reference's 3D zeta flux slot holds, for a node's lower partners, the eta flux between the
        // partner and the last node of its eta line (:702), zero on that node itself
        const bool eta = REF && DIM == 3 && dir == 2;
        double qg[NP][NQ];
        if constexpr (REF && DIM == 3) {
#pragma unroll
            for (int i = 0; i < NP; ++i)
#pragma unroll
                for (int k = 0; k < NQ; ++k) qg[i][k] = q[i][k];
            if (ok && eta) {
#pragma unroll
                for (int i = 0; i < NP - 1; ++i) {
#pragma unroll
                    for (int k = 0; k < NQ; ++k) qg[i][k] = sH[k * ROW + ln % NP + L::SY * (NP - 1) + i * st];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const double x = q[i][k * (1 + DIM)], y = qg[i][k * (1 + DIM)], d = y - x, s = y + x;
                        far = far || !(d * d < 1e-4 * (s * s));
                    }
                }
            }
        }
        const bool any_far = __any_sync(0xffffffffu, far);
        if (ok) {
#pragma unroll
            for (int i = 0; i < NP; ++i)
#pragma unroll
                for (int f = 0; f < NF; ++f) al[i][f] = 0.0;
            auto pairs = [&](auto near) {
#pragma unroll
                for (int i = 0; i < NP - 1; ++i) {
                    double G[NF];
                    if constexpr (REF && DIM == 3) {
                        if (eta) {
                            const double mg[3] = {sGeo[3], sGeo[4], sGeo[5]};
                            line_flux<DIM, decltype(near)::value>(q[i], qg[i], mg, gm1i, G);
                            if (ln / NP == NP - 1)
#pragma unroll
                                for (int f = 0; f < NF; ++f) G[f] = 0.0;
                        }
                    }
#pragma unroll
                    for (int l = i + 1; l < NP; ++l) {
                        double F[NF];
                        line_flux<DIM, decltype(near)::value>(q[i], q[l], m, gm1i, F);
                        const double dil = T.Dhat2[i * NP + l], dli = T.Dhat2[l * NP + i];
#pragma unroll
                        for (int f = 0; f < NF; ++f) {
                            al[i][f] = fma(-dil, F[f], al[i][f]);
                            al[l][f] = fma(-dli, eta ? G[f] : F[f], al[l][f]);
                        }
                    }
                }
            };
            if (any_far) pairs(std::false_type{});
            else pairs(std::true_type{});
            if constexpr (BLEND) {
                if (alpha != 0.0) {   // first-order FV between the line's nodes (DGSEMIntegrator.cpp:972-1196)
                    double mlen = 0.0;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) mlen = fma(m[d], m[d], mlen);
                    mlen = sqrt_pos(mlen);
#pragma unroll
                    for (int i = 0; i < NP; ++i)
#pragma unroll
                        for (int f = 0; f < NF; ++f) al[i][f] *= 1.0 - alpha;
#pragma unroll
                    for (int i = 0; i < NP - 1; ++i) {
                        double qa[L::K], qb[L::K], F[NF];
#pragma unroll
                        for (int k = 0; k < L::K; ++k) {
                            qa[k] = k < NQ ? q[i][k] : sH[k * ROW + n0 + i * st];
                            qb[k] = k < NQ ? q[i + 1][k] : sH[k * ROW + n0 + (i + 1) * st];
                        }
                        line_face_flux<DIM>(qa, qb, m, mlen, gm1i, P.quirks == 0, true, F);
                        const double wa = alpha / T.w[i], wb = alpha / T.w[i + 1];
#pragma unroll
                        for (int f = 0; f < NF; ++f) {
                            al[i][f] = fma(-wa, F[f], al[i][f]);
                            al[i + 1][f] = fma(wb, F[f], al[i + 1][f]);
                        }
                    }
                }
            }
            // the global operands of the line, all in flight together: the traces
            // beyond its two faces, with their viscous rows, and its own viscous rows
            double s[2][NF], v[NP][NF - 1], vn[2][NF - 1];
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                int2 nb = sNbr[2 * (2 * dir + side)];
                if (BC && nb.x < 0) nb = make_int2(e, 2 * dir + side);   // boundary face: the own trace
                const int dn = nb.y >> 1, in = (nb.y & 1) * (NP - 1);
                int na, nbs, nt;
                line_strides<DIM>(dn, NP, NP * NP, na, nbs, nt);
                const long long g = (long long)nb.x * ND + na * (ln % NP) + nbs * (ln / NP) + in * nt;
#pragma unroll
                for (int f = 0; f < NF; ++f) s[side][f] = ldg_now(a.u + f * Ndof + g);
                if constexpr (NS) {
                    const double *gv = REF ? gface + ((long long)nb.x * (2 * DIM) + nb.y) * ((NF - 1) * NL) + ln
                                           : grad + ((long long)nb.x * DIM + dn) * ((NF - 1) * ND) + in * NL + ln;
#pragma unroll
                    for (int f = 0; f < NF - 1; ++f) vn[side][f] = ldg_now(gv + f * (REF ? NL : ND));
                }
            }
            double vo[2][NF - 1];   // the viscous rows of the line's end nodes
            if constexpr (REF) {
#pragma unroll
                for (int side = 0; side < 2; ++side)
#pragma unroll
                    for (int f = 0; f < NF - 1; ++f)
                        vo[side][f] = ldg_now(gface + (((long long)e * (2 * DIM) + 2 * dir + side) * (NF - 1) + f) * NL + ln);
            }
            if constexpr (NS) {
                const double *gv = grad + ((long long)e * DIM + dir) * ((NF - 1) * ND) + ln;
#pragma unroll
                for (int l = 0; l < NP; ++l)
#pragma unroll
                    for (int f = 0; f < NF - 1; ++f) v[l][f] = ldg_now(gv + f * ND + l * NL);
                // sum_l Dhat(i, l) of the rows
#pragma unroll
                for (int l = 0; l < NP; ++l)
#pragma unroll
                    for (int i = 0; i < NP; ++i)
#pragma unroll
                        for (int f = 1; f < NF; ++f) al[i][f] = fma(T.Dhat[i * NP + l], v[l][f - 1], al[i][f]);
                if constexpr (!REF)
#pragma unroll
                    for (int f = 0; f < NF - 1; ++f) {
                        vo[0][f] = v[0][f];
                        vo[1][f] = v[NP - 1][f];
                    }
            }
            // ---- the line's two faces
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int lf = 2 * dir + side, ie = side * (NP - 1);
                const int2 nb = sNbr[2 * lf];
                if (BC && nb.x < 0) {
                    double face[NF];
                    const double fv0[NF - 1] = {};
                    line_boundary<DIM, NS>(a, P, nb.y, sNor + lf * (DIM + 1), s[side], NS ? vo[side] : fv0, side, face);
#pragma unroll
                    for (int f = 0; f < NF; ++f) al[ie][f] = fma(rw0, face[f], al[ie][f]);
                } else {
                    double nor[DIM], qn[L::K], qo[L::K], qa[L::K], qb[L::K], F[NF];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) nor[d] = sNor[lf * (DIM + 1) + d];
                    if constexpr (REF) {
                        // Q8 (BasicOperations.cpp:33-34 via NavierStokesFlux.cpp:14): the surface flux reads
                        // states whose momentum slots hold velocities
                        double so[NF];
                        const double rn = rcp(s[side][0]);
#pragma unroll
                        for (int d = 0; d < DIM; ++d) s[side][1 + d] *= rn;
                        line_prim<DIM>(s[side], gamma, gm1, qn);
                        double vv = 0.0;
                        so[0] = sH[n0 + ie * st];
#pragma unroll
                        for (int d = 0; d < DIM; ++d) {
                            so[1 + d] = sH[(L::V + d) * ROW + n0 + ie * st];
                            vv = fma(so[1 + d], so[1 + d], vv);
                        }
                        // E = p / (gamma - 1) + rho |v|^2 / 2 with p = rho / (2 beta)
                        so[NF - 1] = 0.5 * so[0] * fma(gm1i, sH[L::RBETA * ROW + n0 + ie * st], vv);
                        line_prim<DIM>(so, gamma, gm1, qo);
                    } else {
                        line_prim<DIM>(s[side], gamma, gm1, qn);
#pragma unroll
                        for (int k = 0; k < L::K; ++k) qo[k] = sH[k * ROW + n0 + ie * st];
                    }
                    // both elements evaluate the face with the operands in Elem1, Elem2 order
                    const bool first = sNbr[2 * lf + 1].y == 0;
#pragma unroll
                    for (int k = 0; k < L::K; ++k) {
                        qa[k] = first ? qo[k] : qn[k];
                        qb[k] = first ? qn[k] : qo[k];
                    }
                    line_face_flux<DIM>(qa, qb, nor, sNor[lf * (DIM + 1) + DIM], gm1i, quirk3, P.dissipation != 0, F);
                    const double sg = first ? -rw0 : rw0;
#pragma unroll
                    for (int f = 0; f < NF; ++f) al[ie][f] = fma(sg, F[f], al[ie][f]);
                    if constexpr (NS) {
                        // 0.5 (Fv1 + Fv2) . n: for affine elements the outward scaled normal of local
                        // face lf is (lf odd ? +1 : -1) times row lf/2 of adj(J)
                        const double so = side ? 0.5 * rw0 : -0.5 * rw0, sn = (nb.y & 1) ? -0.5 * rw0 : 0.5 * rw0;
#pragma unroll
                        for (int f = 1; f < NF; ++f)
                            al[ie][f] = fma(so, vo[side][f - 1], fma(sn, vn[side][f - 1], al[ie][f]));
                    }
                }
            }
            // ---- hand the sums on to the next direction's lines
            if (dir > 0) {
#pragma unroll
                for (int i = 0; i < NP; ++i)
#pragma unroll
                    for (int f = 0; f < NF; ++f) al[i][f] += sA[f * ROW + n0 + i * st];
            }
            if (dir < DIM - 1) {
#pragma unroll
                for (int i = 0; i < NP; ++i)
#pragma unroll
                    for (int f = 0; f < NF; ++f) sA[f * ROW + n0 + i * st] = al[i][f];
            }
        }
        if (dir < DIM - 1) sync();
    }
    if (!ok) return;

    // ---- epilogue: the last direction's lines hold the nodes ln, ln + NL, ...
    const double mJ = rcp(sGeo[DIM * DIM]);
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
        for (int f = 0; f < NF; ++f) al[i][f] *= mJ;
    rk_epilogue<NP, NF>(a, al, e0 + ln, NL);
}


// ------------------------------------------------------------ BR1 lifting
// The lifting of the Navier-Stokes form with contravariant viscous fluxes, by
// lines as above: a lane differentiates its line's entropy variables and adds
// the line's two face jumps; the nodes' lanes (the lines of the last direction)
// form the primitive gradients and the viscous rows.  The entropy variables are
// relative to the element's node 0 (constants drop out of derivatives and
// jumps), so that the logarithms are of ratios near one, by series.  The
// node-by-node form (lift_element) spent 30 % of its FP64 instructions on
// logarithms, left half of the threads idle on every second face item and read
// every node's variables 3 Np times; it was bound by latency and barriers at
// 19 warps per SM.  Measured: 32^3 Np = 4 179 -> 109 us (HBM floor 43 us for
// 285 MB), 20^3 Np = 5 90 -> 65 us, 2D 120x60 Np = 5 unchanged at 17 us; in the
// FP32-bulk form, the classes of a 96-member ensemble, 91 -> 48 us (Np = 3),
// 123 -> 70 us (4), 363 -> 231 us (5) and 316 -> 261 us (6).
template <int DIM, int NP, typename W>
struct LiftLineShape : LineShape<DIM, NP, W> {
    using L = LineShape<DIM, NP, W>;
    // rows: entropy variables [NF], derivatives along the first DIM-1 directions [DIM-1][NF];
    // then the neighbour table (two ints a face), adj(J) and 1 / det J
    static constexpr int NBR = DIM * L::NF * L::ROW, GEO = NBR + 4 * DIM * 4 / (int)sizeof(W);
    static constexpr int PER_ELEM = L::padded(GEO + DIM * DIM + 1);
    static_assert((GEO - NBR) * sizeof(W) >= 4 * DIM * sizeof(int) && GEO + DIM * DIM + 1 <= PER_ELEM, "an element's shared area");
    static_assert(sizeof(W) * L::EPB * PER_ELEM + CTX_RESERVE <= MAX_SMEM, "a CTA's shared memory");
};
// D(i, l) in the working precision.
template <typename W>
struct LineD {
    W d[36];
};

// ln(x / x0) for x0 > 0; NaN for x < 0 (u > 1 there: the logarithm).
__device__ __forceinline__ double log_ratio(double x, double x0) {
    const double f = (x - x0) * rcp(x + x0), u = f * f;
    double q = 1.0 / 11.0;
#pragma unroll
    for (int k = 9; k >= 1; k -= 2) q = fma(q, u, 1.0 / k);   // truncation u^6/13 < 1e-19
    if (!(u < 1e-3)) q = log_q_far(x0, x, f, u);
    return 2.0 * f * q;
}
// Entropy variables (BasicOperations.cpp:81-104) of state s relative to those of
// the reference node (rho, p, beta = rho/p, beta |v|^2 / 2).
struct LineRef {
    double rho, p, beta, bvsq;
};
template <int DIM>
__device__ __forceinline__ LineRef line_ref(const double *s, const PhysParams &P) {
    const double r = rcp(s[0]);
    double mm = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) mm = fma(s[1 + d], s[1 + d], mm);
    LineRef R;
    R.rho = s[0];
    R.p = P.gammaM1 * fma(-0.5 * mm, r, s[1 + DIM]);
    R.beta = s[0] * rcp(R.p);
    R.bvsq = R.beta * (0.5 * mm * r * r);
    // a reference node without entropy variables leaves the others theirs, and
    // log_ratio needs a positive one: absolute values then
    if (!(s[0] > 0.0 && R.beta > 0.0 && R.beta < 1e300)) R = LineRef{1.0, 1.0, 0.0, 0.0};
    return R;
}
template <int DIM>
__device__ __forceinline__ void line_entropy(const double *s, const PhysParams &P, const LineRef &R, double *v) {
    const double r = rcp(s[0]);
    double vel[DIM], vv = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        vel[d] = s[1 + d] * r;
        vv = fma(vel[d], vel[d], vv);
    }
    const double p = P.gammaM1 * fma(-0.5 * s[0], vv, s[1 + DIM]);
    const double beta = s[0] * rcp(p);
    const double ds = fma(-P.gamma, log_ratio(s[0], R.rho), log_ratio(p, R.p));
    v[0] = -fma(ds, P.gammaM1Inverse, fma(0.5 * beta, vv, -R.bvsq));
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[1 + d] = beta * vel[d];
    v[1 + DIM] = R.beta - beta;
}
// FP32-bulk form: the same with the logarithms of FP64-formed ratios in FP32.
template <int DIM>
__device__ __forceinline__ void line_entropy(const double *s, const PhysParams &P, const EntropyRef &R, float *v) {
    conserv2entropy_rel<DIM>(s, P, R, v);
}
// The lifting's boundary value minus the inner trace's, as boundary_lift_trace
// defines it (fixed mode): 1/2 (v(outer) - v1), at the no-slip walls v_wall - v1.
template <int DIM>
__device__ __noinline__ void line_lift_boundary(const BcDev &bc, const PhysParams &P, const double *s1,
                                                const double *nor, double *lf) {
    constexpr int NF = DIM + 2;
    double v1[NF];
    conserv2entropy<DIM, double>(s1, P, v1);
    if (bc.type == BC_NOSLIP_ADIABATIC || bc.type == BC_NOSLIP_ISOTHERMAL) {
        const bool adiab = bc.type == BC_NOSLIP_ADIABATIC;
        const double b = adiab ? -v1[NF - 1] : bc.vT;
        lf[0] = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) lf[1 + d] = bc.wall_vel[d] * b - v1[1 + d];
        lf[NF - 1] = adiab ? 0.0 : -bc.vT - v1[NF - 1];
        return;
    }
    double c[NF], s2[NF], v2[NF], nn = 0.0;
#pragma unroll
    for (int f = 0; f < NF; ++f) c[f] = s1[f];
#pragma unroll
    for (int d = 0; d < DIM; ++d) nn += nor[d] * nor[d];
    bc_outer_state<DIM>(bc, c, nor, sqrt(nn), P, s2);
    conserv2entropy<DIM, double>(s2, P, v2);
#pragma unroll
    for (int f = 0; f < NF; ++f) lf[f] = 0.5 * (v2[f] - v1[f]);
}

// REF (reference mode): the rows of the volume term take the state of the
// element's last node (Q1), and the face nodes' own rows follow the volume rows
// of all elements, [E][2 DIM][NF-1][face node].
template <int DIM, int NP, bool BC, bool REF, typename W, typename Sync>
__device__ __forceinline__ void lift_line_element(const ElemIO &a, const PhysParams &P, const LineD<W> &T, double w0, int e,
                                                  bool ok, W *sV, int ln, const Sync &sync) {
    using L = LiftLineShape<DIM, NP, W>;
    constexpr int ND = L::ND, NL = L::NL, NF = L::NF, ROW = L::ROW;
    constexpr bool F64 = sizeof(W) == 8;
    W *sG = sV + NF * ROW, *sGeo = sV + L::GEO;
    int *sNbr = reinterpret_cast<int *>(sV + L::NBR);
    const long long Ndof = a.Ndof, e0 = (long long)e * ND;
    const int own0 = ln % NP + L::SY * (DIM == 2 ? 0 : ln / NP);
    constexpr int own_st = DIM == 2 ? L::SY : L::SZ;
    std::conditional_t<F64, LineRef, EntropyRef> R{};
    if (ok) {
        constexpr int NG = (DIM * DIM + NL) / NL, NB = (2 * DIM + NL - 1) / NL;
        int4 nb[NB];
        double g[NG], s[NP][NF], s0[NF];
#pragma unroll
        for (int k = 0; k < NB; ++k)
            nb[k] = __ldg(a.nbr + (long long)e * (2 * DIM) + min(ln + k * NL, 2 * DIM - 1));
#pragma unroll
        for (int f = 0; f < NF; ++f) s0[f] = __ldg(a.u + f * Ndof + e0);
#pragma unroll
        for (int i = 0; i < NP; ++i)
#pragma unroll
            for (int f = 0; f < NF; ++f) s[i][f] = __ldg(a.u + f * Ndof + e0 + ln + NL * i);
#pragma unroll
        for (int k = 0; k < NG; ++k) g[k] = __ldg(a.geo + (long long)e * (DIM * DIM + 1) + min(ln + k * NL, DIM * DIM));
#pragma unroll
        for (int k = 0; k < NB; ++k)
            if (ln + k * NL < 2 * DIM) {   // element and its local face, or face id and ~(boundary condition)
                sNbr[2 * (ln + k * NL)] = nb[k].x >= 0 ? nb[k].x : nb[k].z;
                sNbr[2 * (ln + k * NL) + 1] = nb[k].x >= 0 ? nb[k].y : ~nb[k].y;
            }
#pragma unroll
        for (int k = 0; k < NG; ++k)
            if (ln + k * NL < DIM * DIM + 1) sGeo[ln + k * NL] = W(ln + k * NL < DIM * DIM ? g[k] : rcp(g[k]));
        if constexpr (F64) R = line_ref<DIM>(s0, P);
        else R = entropy_ref<DIM>(s0, P);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            W v[NF];
            line_entropy<DIM>(s[i], P, R, v);
#pragma unroll
            for (int f = 0; f < NF; ++f) sV[f * ROW + own0 + i * own_st] = v[f];
        }
    }
    sync();

    const W hw0 = W(0.5 / w0);
    W gl[NP][NF];
#pragma unroll 1
    for (int dir = 0; dir < DIM; ++dir) {
        if (ok) {
            int sa, sb, st, ga, gb, gt;
            line_strides<DIM>(dir, L::SY, L::SZ, sa, sb, st);
            line_strides<DIM>(dir, NP, NP * NP, ga, gb, gt);
            const int n0 = sa * (ln % NP) + sb * (ln / NP);
            // neighbour traces of the line's faces (boundary faces: the own trace)
            double s[2][NF];
            int2 nb[2];
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                nb[side] = make_int2(sNbr[2 * (2 * dir + side)], sNbr[2 * (2 * dir + side) + 1]);
                long long g = e0 + ga * (ln % NP) + gb * (ln / NP) + side * (NP - 1) * gt;
                if (!BC || nb[side].y >= 0) {
                    int na, nbs, nt;
                    line_strides<DIM>(nb[side].y >> 1, NP, NP * NP, na, nbs, nt);
                    g = (long long)nb[side].x * ND + na * (ln % NP) + nbs * (ln / NP) + (nb[side].y & 1) * (NP - 1) * nt;
                }
#pragma unroll
                for (int f = 0; f < NF; ++f) s[side][f] = ldg_now(a.u + f * Ndof + g);
            }
            // derivative along the line: sum_l D(i, l) v_l
            W v0[NF], v1[NF];
#pragma unroll
            for (int l = 0; l < NP; ++l) {
                W v[NF];
#pragma unroll
                for (int f = 0; f < NF; ++f) v[f] = sV[f * ROW + n0 + l * st];
#pragma unroll
                for (int i = 0; i < NP; ++i)
#pragma unroll
                    for (int f = 0; f < NF; ++f) gl[i][f] = l == 0 ? T.d[i * NP] * v[f] : fma(T.d[i * NP + l], v[f], gl[i][f]);
                if (l == 0)
#pragma unroll
                    for (int f = 0; f < NF; ++f) v0[f] = v[f];
                if (l == NP - 1)
#pragma unroll
                    for (int f = 0; f < NF; ++f) v1[f] = v[f];
            }
            // + 1/(w0 J) 1/2 (v_neighbour - v_own) n at the ends (LiftingBR1.cpp:10-115); the outward
            // scaled normal of an affine element's local face lf is (lf odd ? +1 : -1) times row lf/2 of
            // adj(J), so the jump adds to the derivative along that row's direction
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                W vn[NF], jump[NF];
                if (BC && nb[side].y < 0) {
                    double in[NF], nor[DIM], lf[NF];
#pragma unroll
                    for (int f = 0; f < NF; ++f) in[f] = s[side][f];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) nor[d] = __ldg(a.fnor + (long long)nb[side].x * DIM + d);
                    line_lift_boundary<DIM>(a.bcs[~nb[side].y], P, in, nor, lf);
#pragma unroll
                    for (int f = 0; f < NF; ++f) jump[f] = W(2.0 * lf[f]);
                } else {
                    line_entropy<DIM>(s[side], P, R, vn);
#pragma unroll
                    for (int f = 0; f < NF; ++f) jump[f] = vn[f] - (side ? v1[f] : v0[f]);
                }
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    if (side) gl[NP - 1][f] = fma(hw0, jump[f], gl[NP - 1][f]);
                    else gl[0][f] = fma(-hw0, jump[f], gl[0][f]);
                }
            }
            if (dir < DIM - 1) {
                W *out = sG + dir * NF * ROW + n0;
#pragma unroll
                for (int i = 0; i < NP; ++i)
#pragma unroll
                    for (int f = 0; f < NF; ++f) out[f * ROW + i * st] = gl[i][f];
            }
        }
    }
    sync();
    if (!ok) return;

    // ---- node by node: gradients (grad1 adj / J, LiftingBR1.cpp:205-206), the chain rule
    // and the contravariant viscous flux adj Fv^T, rows f = 1..NF-1, in line order
    const W mJ = sGeo[DIM * DIM];
    W *gout = reinterpret_cast<W *>(a.grad) + (long long)e * (DIM * (NF - 1) * ND);
    W adj[DIM][DIM];
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int q = 0; q < DIM; ++q) adj[r][q] = sGeo[r * DIM + q];
    W last[3 + DIM];   // REF: rho, 1/rho, v, p of the element's last node
    if constexpr (REF) {
        double s[NF], vv = 0.0;
#pragma unroll
        for (int f = 0; f < NF; ++f) s[f] = __ldg(a.u + f * Ndof + e0 + ND - 1);
        const double rr = rcp(s[0]);
        last[0] = s[0];
        last[1] = rr;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            last[2 + d] = s[1 + d] * rr;
            vv = fma(s[1 + d], s[1 + d], vv);
        }
        last[2 + DIM] = P.gammaM1 * fma(-0.5 * rr, vv, s[NF - 1]);
    }
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int n = own0 + i * own_st;
        double s[NF];
        W sw[NF], g1[DIM][NF], g[DIM][NF], vel[DIM], Vc[DIM][NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            s[f] = __ldg(a.u + f * Ndof + e0 + ln + NL * i);
            sw[f] = W(s[f]);
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
#pragma unroll
            for (int r = 0; r < DIM - 1; ++r) g1[r][f] = sG[(r * NF + f) * ROW + n];
            g1[DIM - 1][f] = gl[i][f];
        }
#pragma unroll
        for (int q = 0; q < DIM; ++q) {
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                W x = g1[0][f] * adj[0][q];
#pragma unroll
                for (int r = 1; r < DIM; ++r) x = fma(g1[r][f], adj[r][q], x);
                g[q][f] = x * mJ;
            }
            entropygrad2primgrad<DIM, W>(sw, P, g[q]);
        }
        // the node's velocity and pressure, formed in FP64
        const double rr = rcp(s[0]);
        double vv = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            vel[d] = W(s[1 + d] * rr);
            vv = fma(s[1 + d], s[1 + d], vv);
        }
        const double p = P.gammaM1 * fma(-0.5 * rr, vv, s[NF - 1]);
        auto rows = [&](W rho, W rrho, const W *vl, W pr) {
#pragma unroll
            for (int r = 0; r < DIM; ++r)
#pragma unroll
                for (int f = 0; f < NF; ++f) Vc[r][f] = 0;
            viscous_flux<DIM, W>(rho, rrho, vl, pr, g, P, [&](int f, int cc, W val) {
#pragma unroll
                for (int r = 0; r < DIM; ++r) Vc[r][f] = fma(adj[r][cc], val, Vc[r][f]);
            });
        };
        rows(sw[0], W(rr), vel, W(p));
        const int c[3] = {ln % NP, DIM == 2 ? i : ln / NP, i};
        if constexpr (REF) {
#pragma unroll
            for (int r = 0; r < DIM; ++r) {
                const int lf = c[r] == 0 ? 2 * r : c[r] == NP - 1 ? 2 * r + 1 : -1;
                if (lf >= 0) {
                    W *out = reinterpret_cast<W *>(a.grad) + Ndof * (DIM * (NF - 1)) +
                             ((long long)e * (2 * DIM) + lf) * ((NF - 1) * NL) + face_tangential<DIM, NP>(r, c);
#pragma unroll
                    for (int f = 1; f < NF; ++f) out[(f - 1) * NL] = Vc[r][f];
                }
            }
            rows(W(last[0]), W(last[1]), last + 2, W(last[2 + DIM]));
        }
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
            W *out = gout + r * (NF - 1) * ND + c[r] * NL + line_index<DIM, NP>(r, c);
#pragma unroll
            for (int f = 1; f < NF; ++f) out[(f - 1) * ND] = Vc[r][f];
        }
    }
}

// A thread's element (slot el of the CTA, mesh element e) and line.
template <typename L>
struct LineLane {
    int el, ln, e;
    bool lane_ok;
    __device__ __forceinline__ LineLane() {
        const int x = L::WARP ? threadIdx.x & 31 : threadIdx.x;
        el = x / L::NL;
        ln = x - el * L::NL;
        lane_ok = el < (L::WARP ? L::EPW : L::EPB);
        if (!lane_ok) el = 0;
        if (L::WARP) el += (threadIdx.x >> 5) * L::EPW;
        e = blockIdx.x * (L::WARP ? (blockDim.x >> 5) * L::EPW : L::EPB) + el;
    }
};
template <typename L>
struct LineSync {
    __device__ __forceinline__ void operator()() const {
        if constexpr (L::WARP) __syncwarp();
        else __syncthreads();
    }
};

// One-shot kernels.  blockDim may be any multiple of 32 up to THREADS when
// elements are packed into warps, THREADS otherwise.
template <int DIM, int NP, bool NS, bool BLEND, bool BC, bool REF>
__global__ void __launch_bounds__(LineShape<DIM, NP>::THREADS, (line_min_blocks<DIM, NP, NS>()))
rhs_line_kernel(const MeshDev m, const RhsArgs a, const PhysParams P, const __grid_constant__ OpTables T) {
    using L = RhsLineShape<DIM, NP>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const LineLane<L> q;
    const bool ok = q.lane_ok && q.e < m.E;
    double *sH = reinterpret_cast<double *>(smem_raw) + q.el * L::PER_ELEM;
    const ElemIO io = io_from_args(m, a);
    rhs_line_element<DIM, NP, NS, BLEND, BC, REF>(io, P, T, ok ? q.e : 0, ok, sH, q.ln, LineSync<L>{});
}
template <int DIM, int NP, bool BC, bool REF, typename W>
__global__ void __launch_bounds__(LineShape<DIM, NP, W>::THREADS, (lift_line_min_blocks<DIM, NP, W>()))
lift_line_kernel(const MeshDev m, const LiftArgs a, const PhysParams P, const __grid_constant__ LineD<W> T, double w0) {
    using L = LiftLineShape<DIM, NP, W>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const LineLane<L> q;
    const bool ok = q.lane_ok && q.e < m.E;
    W *sV = reinterpret_cast<W *>(smem_raw) + q.el * L::PER_ELEM;
    RhsArgs r{};
    r.u = a.u;
    r.grad = a.grad;
    r.grad32 = a.grad32;
    const ElemIO io = io_from_args(m, r);
    lift_line_element<DIM, NP, BC, REF, W>(io, P, T, w0, ok ? q.e : 0, ok, sV, q.ln, LineSync<L>{});
}

// Persistent batch kernel: a fixed grid walks the class's work items, each the
// elements of one warp (or, packed into CTAs, of one CTA) of one solve.  A
// solve's element range is padded to BATCH_CHUNK in the class prefix; every
// chunk holds ceil(BATCH_CHUNK / EPI) items, the last one shorter.  FEAT: the
// class's solves have blending or boundary conditions.
template <typename L, typename W, typename Element>
__device__ __forceinline__ void line_batch_items(const BatchClassDev &c, const BatchStage &st, const Element &element) {
    constexpr int EPI = L::WARP ? L::EPW : L::EPB;                 // elements per item
    constexpr int IPC = (BATCH_CHUNK + EPI - 1) / EPI;             // items per chunk
    constexpr int SLOTS = L::WARP ? L::THREADS / 32 : 1;           // items in flight per CTA
    static_assert(SLOTS * sizeof(WarpCtx) <= CTX_RESERVE, "per-item contexts exceed the reserve");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int slot = L::WARP ? threadIdx.x >> 5 : 0, il = L::WARP ? threadIdx.x & 31 : threadIdx.x;
    WarpCtx *ctx = reinterpret_cast<WarpCtx *>(smem_raw) + slot;
    const int el = il / L::NL, ln = il - el * L::NL;
    const bool lane_ok = el < EPI;
    W *sH = reinterpret_cast<W *>(smem_raw + CTX_RESERVE) + (slot * EPI + (lane_ok ? el : 0)) * L::PER_ELEM;
    const LineSync<L> sync{};
    const int n = c.hdr[0];
    const int total = n > 0 ? c.prefix[n] / BATCH_CHUNK * IPC : 0;
    for (int item = blockIdx.x * SLOTS + slot; item < total; item += gridDim.x * SLOTS) {
        const int chunk = item / IPC, first = chunk * BATCH_CHUNK, in = (item - chunk * IPC) * EPI;
        const int s = batch_slot(c.prefix, n, first);
        BatchInst *Im = c.tab + __ldg(c.ids + s);
        const int E = Im->E;
        const int e0 = first - __ldg(c.prefix + s) + in;
        if (e0 >= E || Im->steps_left <= 0) continue;   // uniform over the item's lanes
        sync();   // the previous item's reads of ctx are done
        {
            const int *src = reinterpret_cast<const int *>(&Im->P);
            int *dst = reinterpret_cast<int *>(&ctx->P);
            if (il < 32)
                for (int q = il; q < (int)(sizeof(PhysParams) / 4); q += 32) dst[q] = src[q];
            if (il == 0) ctx->io = io_from_batch(*Im, Im, st);
        }
        sync();
        const bool ok = lane_ok && e0 + el < E && in + el < BATCH_CHUNK;
        element(ctx->io, ctx->P, ok ? e0 + el : e0, ok, sH, ln, sync);
    }
}
template <int DIM, int NP, bool NS, bool FEAT, int V>
__global__ void __launch_bounds__(LineShape<DIM, NP>::THREADS, (line_min_blocks<DIM, NP, NS, V>()))
rhs_line_batch_kernel(const BatchClassDev c, const BatchStage st, const __grid_constant__ OpTables T) {
    using L = RhsLineShape<DIM, NP>;
    line_batch_items<L, double>(c, st, [&](const ElemIO &io, const PhysParams &P, int e, bool ok, double *sH, int ln,
                                   const LineSync<L> &sync) {
        rhs_line_element<DIM, NP, NS, FEAT, FEAT, false>(io, P, T, e, ok, sH, ln, sync);
    });
}
template <int DIM, int NP, bool FEAT, typename W>
__global__ void __launch_bounds__(LineShape<DIM, NP, W>::THREADS, (lift_line_min_blocks<DIM, NP, W>()))
lift_line_batch_kernel(const BatchClassDev c, const BatchStage st, const __grid_constant__ LineD<W> T, double w0) {
    using L = LiftLineShape<DIM, NP, W>;
    line_batch_items<L, W>(c, st, [&](const ElemIO &io, const PhysParams &P, int e, bool ok, W *sV, int ln,
                                      const LineSync<L> &sync) {
        lift_line_element<DIM, NP, FEAT, false, W>(io, P, T, w0, e, ok, sV, ln, sync);
    });
}
template <typename L>
cudaError_t line_batch_prepare(const void *k, size_t smem, BatchKernelInfo *info) {
    cudaError_t err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    int nb = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, L::THREADS, smem);
    if (err != cudaSuccess) return err;
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, k);
    info->blocks_per_sm = nb;
    info->threads = L::THREADS;
    info->smem = (int)smem;
    info->regs = fa.numRegs;
    info->elems_per_item = L::WARP ? L::EPW : L::EPB;
    return cudaSuccess;
}
template <typename L>
constexpr size_t line_batch_smem() { return CTX_RESERVE + (size_t)L::BYTES * L::EPB * L::PER_ELEM; }
template <typename L, typename Kernel, typename... Args>
cudaError_t line_launch(Kernel k, std::atomic<unsigned> &smem_set, cudaStream_t s, const MeshDev &m, const Args &...args) {
    int threads = L::THREADS;
    if constexpr (L::WARP)   // small meshes: one-warp CTAs, so that every SM gets work
        while (threads > 32 && m.E < 148 * (threads / 32) * L::EPW) threads /= 2;
    const int epb = L::WARP ? threads / 32 * L::EPW : L::EPB;
    const size_t sm = (size_t)L::BYTES * epb * L::PER_ELEM;
    for (int attempt = 0; attempt < 2; ++attempt) {
        cudaError_t err = smem_attribute_once((const void *)k, L::BYTES * L::EPB * L::PER_ELEM, smem_set);
        if (err != cudaSuccess) return err;
        k<<<(m.E + epb - 1) / epb, threads, sm, s>>>(m, args...);
        err = cudaGetLastError();
        if (!smem_attribute_lost(err, sm, smem_set)) return err;
    }
    return cudaErrorInvalidValue;
}
template <int DIM, int NP, bool NS, bool BLEND, bool BC, bool REF = false>
cudaError_t rhs_line_launch(const MeshDev &m, const RhsArgs &a, const PhysParams &P, const OpTables &T, cudaStream_t s) {
    static std::atomic<unsigned> smem_set{0u};
    return line_launch<RhsLineShape<DIM, NP>>(rhs_line_kernel<DIM, NP, NS, BLEND, BC, REF>, smem_set, s, m, a, P, T);
}
template <int NP, typename W>
LineD<W> line_d(const OpTables &T) {
    LineD<W> D{};
    for (int q = 0; q < NP * NP; ++q) D.d[q] = W(T.D[q]);
    return D;
}
template <int DIM, int NP, bool BC, typename W, bool REF = false>
cudaError_t lift_line_launch(const MeshDev &m, const LiftArgs &a, const PhysParams &P, const OpTables &T, cudaStream_t s) {
    static std::atomic<unsigned> smem_set{0u};
    return line_launch<LiftLineShape<DIM, NP, W>>(lift_line_kernel<DIM, NP, BC, REF, W>, smem_set, s, m, a, P, line_d<NP, W>(T), T.w[0]);
}
template <int DIM, int NP, bool NS>
cudaError_t rhs_line_any(const MeshDev &m, const RhsArgs &a, const PhysParams &P, const OpTables &T, cudaStream_t s) {
    if (P.blending)
        return m.bcs ? rhs_line_launch<DIM, NP, NS, true, true>(m, a, P, T, s)
                     : rhs_line_launch<DIM, NP, NS, true, false>(m, a, P, T, s);
    return m.bcs ? rhs_line_launch<DIM, NP, NS, false, true>(m, a, P, T, s)
                 : rhs_line_launch<DIM, NP, NS, false, false>(m, a, P, T, s);
}

}   // namespace
}   // namespace prandtl
