// eval_fp64.cu -- all-FP64 rule evaluation: the plain FP64 form of the engine.
//
// A block evaluates one work item: it cuts a selected parent region along its split
// dimension (cut_region, src/hcubature.cpp:206-218) and applies the Genz-Malik 7/5 rule to
// both children (rule75genzmalik_evalError, src/hcubature.cpp:456-577), or evaluates a
// root region.
// The per-dimension coordinate variants (c, c-+lambda*h) are computed once per child
// together with everything that depends on one coordinate only (10^x, aperture filter,
// HOD occupations, bin indices), then what depends on a few coordinates once per
// projection of the points onto them; each lane then evaluates whole points.  The rule
// sums are formed in the reference's summation order.  Compiled with -fmad=false so every
// product and sum rounds as in the reference's CPU build.
#include "phys64.cuh"

namespace g3l {

struct Slot64 {
    double a[6];
    int i0, i1;
};

// coordinate variant v (0 c, 1/2 c -+ r2, 3/4 c -+ r4, 5/6 c -+ r5) of centre c, half-width hw
__device__ __forceinline__ double variant_x(double c, double hw, int v)
{
    double x = c;
    if (v > 0) {
        double lam = (v <= 2) ? G3L_LAMBDA2 : (v <= 4 ? G3L_LAMBDA4 : G3L_LAMBDA5);
        double rr = hw * lam;
        x = (v & 1) ? c - rr : c + rr;
    }
    return x;
}

// truncated z bin of z = x (the z slot's i1, Model64::fill)
__device__ __forceinline__ int z_trunc64(const DevTables &T, double x)
{
    double zr = ddiv((x - T.zmin) * T.Nz, T.zmax - T.zmin);
    return min(max((int)zr, 0), T.Nz - 1);
}

// An FP64 re-take of an unsettled split (a split-only entry) needs the centre and the axis
// points of the contending dimensions only: cm, the dimensions whose fourth-difference
// bounds reach the leader's (P.cmask, written by the FP32 rule kernel with the flag).  The
// others' differences are below the leader's under those bounds, so the FP64 choice among
// the contenders is the FP64 choice among all dimensions.
__device__ __forceinline__ unsigned split_cmask(const Pool &P, const IntDesc &d, int2 ent)
{
    return (unsigned)P.cmask[d.base + (ent.y & 0x3FFFFFFF)];
}

template <int KIND, int TERM>
struct Model64 {
    static constexpr int DIM = TERM + 4;

    // N_sat pair count of a mass slot: with the rescaling s of the hod1 slot at this mass's
    // rounded bin (src/NNMap_Model.cu:563,808)
    __device__ static double pairs(const DevTables &T, const IntDesc &d, const Slot64 &S)
    {
        return nsatnsat64(S.a[2], S.a[4], d.same, T.A, T.eps, S.a[0],
                          __ldg(T.scale + (size_t)d.hod1 * T.Nm + S.i0));
    }

    // A halo mass's slot without the second population (two populations: S.a[3..5])
    __device__ static void fill_mass(const DevTables &T, const IntDesc &d, double x, Slot64 &S,
                                     unsigned long long *ties)
    {
        const double m = pow(10, x);
        S.a[0] = m;
        m_index(T, x, m, S.i0, S.i1, ties);
        occupations64(T.hod + 6 * d.hod1, m, S.a[1], S.a[2]);
        if (KIND == 0 && d.same) {  // the second population's occupations are the first's
            S.a[3] = S.a[1];
            S.a[4] = S.a[2];
            S.a[5] = pairs(T, d, S);
        }
    }

    // Fill one coordinate-variant slot (everything that depends on one coordinate).
    __device__ static void fill(const DevTables &T, const IntDesc &d, int dimidx, double x,
                                Slot64 &S, unsigned long long *ties)
    {
        if (dimidx < 2) {  // l1, l2 (log10 l)
            double l = pow(10, x);
            S.a[0] = l;
            S.a[1] = aperture64(d.theta[dimidx] * l);
        } else if (dimidx == 2) {  // phi
            S.a[0] = cos(x);
        } else if (dimidx < 3 + TERM) {  // halo masses (log10 m)
            fill_mass(T, d, x, S, ties);
            if (KIND == 0 && !d.same) {
                occupations64(T.hod + 6 * d.hod2, S.a[0], S.a[3], S.a[4]);
                S.a[5] = pairs(T, d, S);
            }
        } else {  // z
            S.a[0] = x;
            double zr = ddiv((x - T.zmin) * T.Nz, T.zmax - T.zmin);
            S.i0 = min(max((int)round(zr), 0), T.Nz - 1);
            S.i1 = min(max((int)zr, 0), T.Nz - 1);
        }
    }

    // Integrand at one point from its variant slots (kernel_function_* of the reference).
    // Operands of the shared u_NFW, with the expressions of point(); mz: r_200 and F of the
    // (mass, z) pair.  Cached u_NFW f (ucache_fun) at slots L (l), M (mass), Z (z):
    __device__ static void ucached_args(const DevTables &T, const IntDesc &d, int f, const Slot64 &L,
                                        const Slot64 &M, const Slot64 &Z, const double *mz,
                                        double &k, double &r200, double &c, double &F)
    {
        const double w_ = __ldg(T.w + Z.i0);
        const double conc = __ldg(T.conc + Z.i1 * T.Nm + M.i1);
        const int fs = ucache_fun(KIND, TERM, f, 2);
        k = ddiv(L.a[0], w_);
        r200 = mz[0];
        c = (fs == 0 ? 1.0 : (fs == 1 ? T.hod[6 * d.hod1] : T.hod[6 * d.hod2])) * conc;
        F = mz[1 + fs];
    }

    // u_NFW(k3, mass u3_mass(f)): shared by the points with the same projection (u3_drop)
    __device__ static void u3_args(const DevTables &T, int f, const Slot64 *const *s,
                                   const double *mz, double &k, double &r200, double &c, double &F)
    {
        const Slot64 &L1 = *s[0], &L2 = *s[1], &PH = *s[2], &Z = *s[DIM - 1];
        const Slot64 &M = *s[u3_mass(KIND, TERM, f)];
        const double l1 = L1.a[0], l2 = L2.a[0], cphi = PH.a[0];
        const double w_ = __ldg(T.w + Z.i0);
        const double l3 = sqrt(l1 * l1 + l2 * l2 + 2 * l1 * l2 * cphi);
        k = ddiv(l3, w_);
        r200 = mz[0];
        c = 1.0 * __ldg(T.conc + Z.i1 * T.Nm + M.i1);
        F = mz[1];
    }

    // F at factors 1, f of hod1, f of hod2 (nf of them) of halo mass slot M at z bin zt, with
    // the expressions of point(): o[1..nf]
    __device__ static void mz_norms(const DevTables &T, const IntDesc &d, const Slot64 &M, int zt,
                                    int nf, double *o)
    {
        const double conc = __ldg(T.conc + zt * T.Nm + M.i1);
        double c0 = 0, F = 0;
        for (int q = 0; q < nf; ++q) {
            const double c = (q == 0 ? 1.0 : (q == 1 ? T.hod[6 * d.hod1] : T.hod[6 * d.hod2])) * conc;
            if (q == 0 || c != c0) F = nfw_norm64(c);  // equal factors share it
            c0 = c;
            o[1 + q] = F;
        }
    }

    // r_200 and the normalisations: o[0..nf]
    __device__ static void mz_values(const DevTables &T, const IntDesc &d, const Slot64 &M, int zt,
                                     int nf, double *o)
    {
        o[0] = r200_64(M.a[0], __ldg(T.rho_bar + zt));
        mz_norms(T, d, M, zt, nf, o);
    }

    // auxiliary function a (aux_dims) with the expressions of point(): the aperture filter
    // of l3; P_lin at k1, k2, k3 (2-halo); the tree-level bispectrum (3-halo)
    __device__ static double aux(const DevTables &T, const IntDesc &d, int a, const Slot64 *const *s)
    {
        const Slot64 &L1 = *s[0], &L2 = *s[1], &PH = *s[2];
        const double l1 = L1.a[0], l2 = L2.a[0], cphi = PH.a[0];
        const double l3 = sqrt(l1 * l1 + l2 * l2 + 2 * l1 * l2 * cphi);
        if (a == 0) return aperture64(d.theta[2] * l3);
        const int z_ix = s[DIM - 1]->i0;
        const double w_ = __ldg(T.w + z_ix);
        if (TERM == 3) return bi_lin64(T, ddiv(l1, w_), ddiv(l2, w_), cphi, z_ix);
        return plin64(T, z_ix, ddiv(a == 1 ? l1 : (a == 2 ? l2 : l3), w_));
    }

    // uc: the cached u_NFW values of this point (ucache_fun order), or null; u3c: its
    // cached u_NFW at k3 (u3()), or null; ax: its cached auxiliary values (aux()), or null
    __device__ static double point(const DevTables &T, const IntDesc &d, const Slot64 *const *s,
                                   const double *uc = nullptr, const double *u3c = nullptr,
                                   const double *ax = nullptr)
    {
        const Slot64 &L1 = *s[0], &L2 = *s[1], &PH = *s[2], &Z = *s[DIM - 1];
        const double l1 = L1.a[0], l2 = L2.a[0], cphi = PH.a[0], z = Z.a[0];
        const int z_ix = Z.i0, z_it = Z.i1, Nm = T.Nm;
        const double w_ = __ldg(T.w + z_ix);
        const double l3 = sqrt(l1 * l1 + l2 * l2 + 2 * l1 * l2 * cphi);
        const double k1 = ddiv(l1, w_);
        const double k2 = ddiv(l2, w_);
        const double k3 = ddiv(l3, w_);
        const double rho = __ldg(T.rho_bar + z_ix);
        const double rhot = __ldg(T.rho_bar + z_it);
        const double f1 = T.hod[6 * d.hod1];
        const double U3 = ax ? ax[0] : aperture64(d.theta[2] * l3);
        if (KIND == 0) {
            const double nbar1 = __ldg(T.nbar + d.hod1 * T.Nz + z_ix);
            const double nbar2 = __ldg(T.nbar + d.hod2 * T.Nz + z_ix);
            const double f2 = T.hod[6 * d.hod2];
            if (TERM == 1) {
                // src/NNMap_Model.cu:544-593
                const Slot64 &M = *s[3];
                const double m = M.a[0];
                const double r2 = r200_64(m, rhot);
                const double cc = __ldg(T.conc + z_it * Nm + M.i1);
                const double u3 = u3c ? u3c[0] : u_nfw64(k3, r2, cc, 1);
                const double u2 = uc ? uc[1] : u_nfw64(k2, r2, cc, f2);
                const double u1 = uc ? uc[0] : u_nfw64(k1, r2, cc, f1);
                double Bggd = ddiv(ddiv(ddiv(1., nbar1), nbar2), rho) * __ldg(T.hmf + z_ix * Nm + M.i0) * m * u3;
                Bggd *= M.a[1] * M.a[4] * u2 + M.a[3] * M.a[2] * u1 + M.a[5] * u1 * u2;
                double bggk = ddiv(Bggd, __ldg(T.dwdz + z_ix)) * __ldg(T.g + z_ix) *
                              __ldg(T.p1 + z_ix) * __ldg(T.p2 + z_ix);
                bggk = ddiv(ddiv(ddiv(bggk, w_), w_), w_) * (1. + z);
                return l1 * l2 * m * l1 * l2 * L1.a[1] * L2.a[1] * U3 * bggk;
            } else if (TERM == 2) {
                // src/NNMap_Model.cu:787-856
                const Slot64 &M1 = *s[3], &M2 = *s[4];
                const double m1 = M1.a[0], m2 = M2.a[0];
                const double Pk1 = ax ? ax[1] : plin64(T, z_ix, k1);
                const double Pk2 = ax ? ax[2] : plin64(T, z_ix, k2);
                const double Pk3 = ax ? ax[3] : plin64(T, z_ix, k3);
                const double ra = r200_64(m1, rhot), rb = r200_64(m2, rhot);
                const double ca = __ldg(T.conc + z_it * Nm + M1.i1);
                const double cb = __ldg(T.conc + z_it * Nm + M2.i1);
                const double u3_1 = u3c ? u3c[0] : u_nfw64(k3, ra, ca, 1);
                const double u3_2 = u3c ? u3c[1] : u_nfw64(k3, rb, cb, 1);
                const double u1_1 = uc ? uc[0] : u_nfw64(k1, ra, ca, f1);
                const double u2_1 = uc ? uc[1] : u_nfw64(k2, ra, ca, f2);
                const double u1_2 = uc ? uc[2] : u_nfw64(k1, rb, cb, f1);
                const double u2_2 = uc ? uc[3] : u_nfw64(k2, rb, cb, f2);
                // G_gg(k1, k2, m2)
                const double Ggg = M2.a[1] * M2.a[4] * u2_2 + M2.a[3] * M2.a[2] * u1_2 +
                                   M2.a[5] * u1_2 * u2_2;
                const double Gg_k1m1 = M1.a[1] + M1.a[2] * u1_1;  // hod1 at m1
                const double Gg_k2m2 = M2.a[3] + M2.a[4] * u2_2;  // hod2 at m2
                const double Gg_k2m1 = M1.a[3] + M1.a[4] * u2_1;  // hod2 at m1
                const double Gg_k1m2 = M2.a[1] + M2.a[2] * u1_2;  // hod1 at m2
                double Bggd = ddiv(ddiv(ddiv(1., nbar1), nbar2), rho) * __ldg(T.hmf + z_ix * Nm + M1.i0) *
                              __ldg(T.hmf + z_ix * Nm + M2.i0) * __ldg(T.b_h + z_ix * Nm + M1.i0) *
                              __ldg(T.b_h + z_ix * Nm + M2.i0) *
                              (m1 * u3_1 * Ggg * Pk3 + m2 * u3_2 * Gg_k1m1 * Gg_k2m2 * Pk1 +
                               m2 * u3_2 * Gg_k2m1 * Gg_k1m2 * Pk2);
                double bggk = ddiv(1., __ldg(T.dwdz + z_ix)) * __ldg(T.g + z_ix) *
                              __ldg(T.p1 + z_ix) * __ldg(T.p2 + z_ix);
                bggk = ddiv(ddiv(ddiv(bggk, w_), w_), w_) * (1. + z) * Bggd;
                return l1 * l2 * m1 * m2 * l1 * l2 * L1.a[1] * L2.a[1] * U3 * bggk;
            } else {
                // src/NNMap_Model.cu:1003-1037
                const Slot64 &M1 = *s[3], &M2 = *s[4], &M3 = *s[5];
                const double m1 = M1.a[0], m2 = M2.a[0], m3 = M3.a[0];
                const double u3 = u3c ? u3c[0]
                                      : u_nfw64(k3, r200_64(m3, rhot), __ldg(T.conc + z_it * Nm + M3.i1), 1);
                const double u1 = uc ? uc[0] : u_nfw64(k1, r200_64(m1, rhot), __ldg(T.conc + z_it * Nm + M1.i1), f1);
                const double u2 = uc ? uc[1] : u_nfw64(k2, r200_64(m2, rhot), __ldg(T.conc + z_it * Nm + M2.i1), f2);
                const double Gg1 = M1.a[1] + M1.a[2] * u1;  // hod1 at m1
                const double Gg2 = M2.a[3] + M2.a[4] * u2;  // hod2 at m2
                double Bggd = ddiv(ddiv(ddiv(1., nbar1), nbar2), rho) * __ldg(T.hmf + z_ix * Nm + M1.i0) *
                              __ldg(T.hmf + z_ix * Nm + M2.i0) * __ldg(T.hmf + z_ix * Nm + M3.i0) *
                              m3 * u3 * Gg1 * Gg2 * (ax ? ax[1] : bi_lin64(T, k1, k2, cphi, z_ix)) *
                              __ldg(T.b_h + z_ix * Nm + M1.i0) * __ldg(T.b_h + z_ix * Nm + M2.i0) *
                              __ldg(T.b_h + z_ix * Nm + M3.i0);
                double bggk = ddiv(Bggd, __ldg(T.dwdz + z_ix)) * __ldg(T.g + z_ix) *
                              __ldg(T.p1 + z_ix) * __ldg(T.p2 + z_ix);
                bggk = ddiv(ddiv(ddiv(bggk, w_), w_), w_) * (1. + z);
                return l1 * l2 * m1 * m2 * m3 * l1 * l2 * L1.a[1] * L2.a[1] * U3 * bggk;
            }
        } else {
            const double nbar = __ldg(T.nbar + d.hod1 * T.Nz + z_ix);
            const double f = f1;
            const double gz = __ldg(T.g + z_ix);
            if (TERM == 1) {
                // src/NMapMap_Model.cu:263-301
                const Slot64 &M = *s[3];
                const double m = M.a[0];
                const double r2 = r200_64(m, rhot);
                const double cc = __ldg(T.conc + z_it * Nm + M.i1);
                double Bgdd = ddiv(ddiv(ddiv(1., nbar), rho), rho) * __ldg(T.hmf + z_ix * Nm + M.i0) * m * m *
                              (M.a[1] + M.a[2] * (uc ? uc[0] : u_nfw64(k1, r2, cc, f))) *
                              (uc ? uc[1] : u_nfw64(k2, r2, cc, 1)) *
                              (u3c ? u3c[0] : u_nfw64(k3, r2, cc, 1));
                double bgkk = ddiv(Bgdd, __ldg(T.dwdz + z_ix)) * gz * gz * __ldg(T.p1 + z_ix);
                bgkk = ddiv(ddiv(bgkk, w_), w_) * (1. + z) * (1. + z);
                return ddiv(l1 * l2 * m * l1 * l2 * L1.a[1] * L2.a[1] * U3 * bgkk, nbar);
            } else if (TERM == 2) {
                // src/NMapMap_Model.cu:402-468
                const Slot64 &M1 = *s[3], &M2 = *s[4];
                const double m1 = M1.a[0], m2 = M2.a[0];
                const double Pk1 = ax ? ax[1] : plin64(T, z_ix, k1);
                const double Pk2 = ax ? ax[2] : plin64(T, z_ix, k2);
                const double Pk3 = ax ? ax[3] : plin64(T, z_ix, k3);
                const double ra = r200_64(m1, rhot), rb = r200_64(m2, rhot);
                const double ca = __ldg(T.conc + z_it * Nm + M1.i1);
                const double cb = __ldg(T.conc + z_it * Nm + M2.i1);
                const double u2_1 = uc ? uc[0] : u_nfw64(k2, ra, ca, 1);
                const double u3_2 = u3c ? u3c[1] : u_nfw64(k3, rb, cb, 1);
                const double u1_2f = uc ? uc[1] : u_nfw64(k1, rb, cb, f);
                const double u3_1 = u3c ? u3c[0] : u_nfw64(k3, ra, ca, 1);
                const double u2_2 = uc ? uc[2] : u_nfw64(k2, rb, cb, 1);
                const double u1_1f = uc ? uc[3] : u_nfw64(k1, ra, ca, f);
                double Bgdd = ddiv(ddiv(ddiv(1., nbar), rho), rho) * __ldg(T.hmf + z_ix * Nm + M1.i0) *
                              __ldg(T.hmf + z_ix * Nm + M2.i0) * __ldg(T.b_h + z_ix * Nm + M1.i0) *
                              __ldg(T.b_h + z_ix * Nm + M2.i0) *
                              (m1 * m2 * u2_1 * u3_2 * (M2.a[1] + M2.a[2] * u1_2f) * Pk2 +
                               m1 * m2 * u3_1 * u2_2 * (M2.a[1] + M2.a[2] * u1_2f) * Pk3 +
                               m2 * m2 * u2_1 * u3_2 * (M1.a[1] + M1.a[2] * u1_1f) * Pk1);
                double bgkk = ddiv(Bgdd, __ldg(T.dwdz + z_ix)) * gz * gz * __ldg(T.p1 + z_ix);
                bgkk = ddiv(ddiv(bgkk, w_), w_) * (1. + z) * (1. + z);
                return ddiv(l1 * l2 * m1 * m2 * l1 * l2 * L1.a[1] * L2.a[1] * U3 * bgkk, nbar);
            } else {
                // src/NMapMap_Model.cu:592-632 (Nc, Ns at m3; u_NFW(k1, m2, f))
                const Slot64 &M1 = *s[3], &M2 = *s[4], &M3 = *s[5];
                const double m1 = M1.a[0], m2 = M2.a[0], m3 = M3.a[0];
                const double ra = r200_64(m1, rhot), rb = r200_64(m2, rhot);
                const double ca = __ldg(T.conc + z_it * Nm + M1.i1);
                const double cb = __ldg(T.conc + z_it * Nm + M2.i1);
                double Bgdd = ddiv(ddiv(ddiv(1., nbar), rho), rho) * __ldg(T.hmf + z_ix * Nm + M1.i0) *
                              __ldg(T.hmf + z_ix * Nm + M2.i0) * __ldg(T.hmf + z_ix * Nm + M3.i0) *
                              __ldg(T.b_h + z_ix * Nm + M1.i0) * __ldg(T.b_h + z_ix * Nm + M2.i0) *
                              __ldg(T.b_h + z_ix * Nm + M3.i0) * m1 * m2 *
                              (uc ? uc[0] : u_nfw64(k2, ra, ca, 1)) *
                              (u3c ? u3c[0] : u_nfw64(k3, rb, cb, 1)) *
                              (M3.a[1] + M3.a[2] * (uc ? uc[1] : u_nfw64(k1, rb, cb, f))) *
                              (ax ? ax[1] : bi_lin64(T, k1, k2, cphi, z_ix));
                double bgkk = ddiv(Bgdd, __ldg(T.dwdz + z_ix)) * gz * gz * __ldg(T.p1 + z_ix);
                bgkk = ddiv(ddiv(bgkk, w_), w_) * (1. + z) * (1. + z);
                return ddiv(l1 * l2 * m1 * m2 * m3 * l1 * l2 * L1.a[1] * L2.a[1] * U3 * bgkk, nbar);
            }
        }
    }
};

template <int KIND, int TERM>
__global__ void __launch_bounds__(128) k_re_tables(unsigned char *out)
{
    using RT = ReTab<KIND, TERM>;
    static_assert(sizeof(RT) <= RETAB_BYTES && sizeof(RT) % 4 == 0, "re-evaluation table size");
    __shared__ __align__(16) unsigned char buf[sizeof(RT)];
    __shared__ uint8_t map[RT::NF * 343];
    RT &t = *reinterpret_cast<RT *>(buf);
    ucache_tables<KIND, TERM>(t.ucidx, t.ucl, t.ucn, map);
    for (int p = threadIdx.x; p < RT::NP; p += blockDim.x) t.sdesc[p] = point_variants(RT::DIM, p);
    __syncthreads();
    u3_tables<KIND, TERM>(t.sdesc, t.u3rep, t.u3list, map);  // map is free again
    aux_tables<TERM>(t.sdesc, t.auxrep, t.auxlist, map);
    uint32_t *dst = reinterpret_cast<uint32_t *>(out + (KIND * 3 + TERM - 1) * RETAB_BYTES);
    for (int i = threadIdx.x; i < (int)(sizeof(RT) / 4); i += blockDim.x)
        dst[i] = reinterpret_cast<const uint32_t *>(buf)[i];
}

// Shared memory of one work item.  Child 1 has its own copy of a cached function only when
// the split dimension is among the function's dimensions.
template <int KIND, int TERM>
struct Item64 {
    static constexpr int DIM = TERM + 4, NP = rule_points(DIM), NF = ucache_nf(TERM);
    static constexpr int NU3 = u3_nfun(TERM), NA = aux_nfun(TERM);
    static constexpr int NAUX = aux_off(TERM, NA - 1) + aux_count(TERM, NA - 1);
    Slot64 slots[(DIM + 1) * NVAR];
    double mz[2][TERM][MZ_PAIRS][MZ_VALS];
    double uc[2][NF][UC_MAX];
    double u3[2][NU3][U3_MAX];
    double aux[2][NAUX];
    double vals[2 * NP];
};

// Rule sums of both children by one warp, each sum in the reference's order
// (src/hcubature.cpp:512-576): eight lanes per child form the axis sums, the pair sum, the
// corner sum and one fourth difference each.  An FP64 instruction occupies the pipe for 64
// cycles however few lanes take part, so the sums run side by side, not one after another.
// Valid in lanes 0 (child 0) and 8 (child 1).
template <int DIM>
__device__ void combine64_warp(const double *v, double vol, double &val, double &err, int &split)
{
    const int r = threadIdx.x & 7;
    const double ratio = (G3L_LAMBDA2 * G3L_LAMBDA2) / (G3L_LAMBDA4 * G3L_LAMBDA4);
    const double weight1 = (double)(12824 - 9120 * DIM + 400 * DIM * DIM) / (double)19683;
    const double weight3 = (double)(1820 - 400 * DIM) / (double)19683;
    const double weight5 = (double)6859 / (double)19683 / (double)(1u << DIM);
    const double weightE1 = (double)(729 - 950 * DIM + 50 * DIM * DIM) / (double)729;
    const double weightE3 = (double)(265 - 100 * DIM) / (double)1458;
    const double weight2 = 980. / 6561., weight4 = 200. / 19683.;
    const double weightE2 = 245. / 486., weightE4 = 25. / 729.;
    constexpr int NRR = 2 * DIM * (DIM - 1), NC = 1 << DIM;
    const double val0 = v[0];
    // lane r = 0, 1: pairs of axis points at lambda2, lambda4; 2: (+-, +-) points; 3: corners
    const double *p = v + (r == 2 ? 1 + 4 * DIM : (r == 3 ? 1 + 4 * DIM + NRR : 1 + 2 * r));
    const int n = r < 2 ? DIM : (r == 2 ? NRR : (r == 3 ? NC : 0));
    double s = 0;
    constexpr int NMAX = NRR > NC ? NRR : NC;
    for (int k = 0; k < NMAX; ++k)
        if (k < n) s += r < 2 ? p[4 * k] + p[4 * k + 1] : p[k];
    // fourth difference of dimension r
    long long db = 0;
    if (r < DIM) {
        const double *q = v + 1 + 4 * r;
        double diff = 0;
        diff += fabs(q[0] + q[1] - 2 * val0 - ratio * (q[2] + q[3] - 2 * val0));
        if (diff > 0) db = __double_as_longlong(diff);  // NaN never exceeds the maximum
    }
    const double sum2 = __shfl_sync(0xffffffffu, s, 0, 8), sum3 = __shfl_sync(0xffffffffu, s, 1, 8);
    const double sum4 = __shfl_sync(0xffffffffu, s, 2, 8), sum5 = __shfl_sync(0xffffffffu, s, 3, 8);
    long long maxdiff = 0;
    int dimDiffMax = 0;
    for (int k = 0; k < DIM; ++k) {  // the first maximum
        const long long o = __shfl_sync(0xffffffffu, db, k, 8);
        if (o > maxdiff) {
            maxdiff = o;
            dimDiffMax = k;
        }
    }
    const double result = vol * (weight1 * val0 + weight2 * sum2 + weight3 * sum3 + weight4 * sum4 +
                                 weight5 * sum5);
    const double res5th =
        vol * (weightE1 * val0 + weightE2 * sum2 + weightE3 * sum3 + weightE4 * sum4);
    val = result;
    err = fabs(res5th - result);
    split = dimDiffMax;
}

// One work item on a block of 128 threads: `cut` = bisect the region at pslot along its split
// dimension into pslot (lower half) and qslot (upper half) and evaluate both; otherwise
// evaluate the region at pslot in place (roots).  Four passes with a barrier between:
// coordinate slots; (mass, z) values and the auxiliary functions; every u_NFW that several
// points share; the points.  A quantity is evaluated once per projection of the rule's
// points onto the dimensions it depends on, and for child 1 only if the split dimension is
// one of them, by the expressions of the per-point code (bit-identical values).  The FP64
// pipe bounds this kernel (one warp instruction per 64 cycles per SM quarter), so what
// counts is the number of warp instructions: the 2-halo rule takes 132 + 186 u_NFW per
// child at most instead of 894, the 3-halo rule 66 + 93 instead of 723.
template <int KIND, int TERM>
__device__ void block_item64(const DevTables &T, const IntDesc &d, const Pool &P, long long pslot,
                             long long qslot, bool cut, Item64<KIND, TERM> &I,
                             const ReTab<KIND, TERM> &tb, int rank, unsigned long long *ties,
                             double *dbg)
{
    using M = Model64<KIND, TERM>;
    using It = Item64<KIND, TERM>;
    constexpr int DIM = It::DIM, NP = It::NP, NF = It::NF, NU3 = It::NU3, NA = It::NA;
    constexpr int ZD = DIM - 1;
    const int lane = threadIdx.x & 31;
    const long long stride = P.stride;
    const int sdim = cut ? P.split[pslot] : 0;
    const int nchild = cut ? 2 : 1;
    double c_l = 0;
    int lev = 0;
    if (lane < DIM) {
        c_l = P.center[lane * stride + pslot];
        lev = P.level[lane * stride + pslot];
    }
    const int levs = __shfl_sync(0xffffffffu, lev, sdim) + (cut ? 1 : 0);
    const double cs = __shfl_sync(0xffffffffu, c_l, sdim);
    double cL = cs, cR = cs;
    if (cut) {
        const double hws = ldexp(d.hw0[sdim], -levs);
        cL = cs - hws;
        cR = cs + hws;
    }
    const int levsum = __reduce_add_sync(0xffffffffu, lane < DIM ? lev : 0) + (cut ? 1 : 0);
    // does child 1 need its own values of a function of the dimensions dims?
    auto own = [&](uint32_t dims) { return cut && ((dims >> sdim) & 1u); };
    // coordinate slots, masses first (the longest path), then l, phi, z: the warps then
    // diverge least.  Slots of child 1's split dimension follow those of its kind.
    {
        const bool smass = cut && sdim >= 3 && sdim < 3 + TERM;
        const int nm = TERM * NVAR, nms = nm + (smass ? NVAR : 0);
        const int nslot = (DIM + nchild - 1) * NVAR;
        for (int t = rank; t < nslot; t += 128) {
            int sd;  // slot row: dimension, or DIM for child 1's split dimension
            if (t < nms) {
                sd = t / NVAR < TERM ? 3 + t / NVAR : DIM;
            } else {
                const int q = (t - nms) / NVAR;
                sd = q < 3 ? q : (q == 3 ? ZD : DIM);
            }
            const int v = t % NVAR, dim = sd < DIM ? sd : sdim;
            int L = P.level[dim * stride + pslot];
            double c = P.center[dim * stride + pslot];
            if (cut && dim == sdim) {
                L += 1;
                c = sd < DIM ? cL : cR;
            }
            M::fill(T, d, dim, variant_x(c, ldexp(d.hw0[dim], -L), v), I.slots[sd * NVAR + v], ties);
        }
    }
    __syncthreads();
    auto slot = [&](int ch, int dim, int v) -> const Slot64 & {
        return I.slots[((ch && dim == sdim) ? DIM : dim) * NVAR + v];
    };
    // r_200 and F per (mass, z) pair; auxiliary functions per projection
    {
        int nmz[TERM], nax[NA], tot = 0;
#pragma unroll
        for (int k = 0; k < TERM; ++k) {
            nmz[k] = MZ_PAIRS * (own((8u << k) | (1u << ZD)) ? 2 : 1);
            tot += nmz[k];
        }
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            nax[a] = aux_count(TERM, a) * (own(aux_dims(TERM, a)) ? 2 : 1);
            tot += nax[a];
        }
        for (int t0 = rank; t0 < tot; t0 += 128) {
            int t = t0, k = 0, a = -1;
#pragma unroll
            for (int q = 0; q < TERM; ++q)
                if (k == q && t >= nmz[q]) {
                    t -= nmz[q];
                    ++k;
                }
            if (k < TERM) {
                const int ch = t >= MZ_PAIRS, j = t - ch * MZ_PAIRS;
                const int vm = mz_vm_of(j), vz = mz_vz_of(j);
                M::mz_values(T, d, slot(ch, 3 + k, vm), slot(ch, ZD, vz).i1, KIND == 0 ? 3 : 2,
                             I.mz[ch][k][j]);
                continue;
            }
            a = 0;
#pragma unroll
            for (int q = 0; q < NA - 1; ++q)
                if (a == q && t >= nax[q]) {
                    t -= nax[q];
                    ++a;
                }
            const int na = aux_count(TERM, a);
            const int ch = t >= na, j = t - ch * na;
            const uint32_t vv = tb.sdesc[tb.auxlist[aux_off(TERM, a) + j]];
            const Slot64 *sp[DIM];
#pragma unroll
            for (int dd = 0; dd < DIM; ++dd) sp[dd] = &slot(ch, dd, (vv >> (3 * dd)) & 7);
            I.aux[ch][aux_off(TERM, a) + j] = M::aux(T, d, a, sp);
        }
    }
    __syncthreads();
    // shared u_NFW: (l, m, z) combinations, then k3 projections
    {
        int nu[NF], n3[NU3], tot = 0;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const uint32_t dims = (1u << ucache_fun(KIND, TERM, f, 0)) |
                                  (1u << ucache_fun(KIND, TERM, f, 1)) | (1u << ZD);
            nu[f] = tb.ucn[f] * (own(dims) ? 2 : 1);
            tot += nu[f];
        }
#pragma unroll
        for (int f = 0; f < NU3; ++f) {
            n3[f] = U3_MAX * (own(7u | (1u << u3_mass(KIND, TERM, f)) | (1u << ZD)) ? 2 : 1);
            tot += n3[f];
        }
        for (int t0 = rank; t0 < tot; t0 += 128) {
            int t = t0, f = 0;
            bool lmz = true;
            double kk, r200, cc, F, *out;
#pragma unroll
            for (int q = 0; q < NF; ++q)
                if (f == q && t >= nu[q]) {
                    t -= nu[q];
                    ++f;
                }
            if (f == NF) {
                lmz = false;
                f = 0;
                if (NU3 == 2 && t >= n3[0]) {
                    t -= n3[0];
                    f = 1;
                }
            }
            if (lmz) {
                const int n = tb.ucn[f], ch = t >= n, j = t - ch * n;
                const uint32_t key = tb.ucl[f * UC_MAX + j];
                const int vl = key & 7, vm = (key >> 3) & 7, vz = (key >> 6) & 7;
                const int dl = ucache_fun(KIND, TERM, f, 0), dm = ucache_fun(KIND, TERM, f, 1);
                const int mc = ch && own((1u << dm) | (1u << ZD));
                M::ucached_args(T, d, f, slot(ch, dl, vl), slot(ch, dm, vm), slot(ch, ZD, vz),
                                I.mz[mc][dm - 3][mz_index(vm, vz)], kk, r200, cc, F);
                out = &I.uc[ch][f][j];
            } else {
                const int ch = t >= U3_MAX, j = t - ch * U3_MAX;
                const uint32_t vv = tb.sdesc[tb.u3list[f * U3_MAX + j]];
                const int dm = u3_mass(KIND, TERM, f);
                const int mc = ch && own((1u << dm) | (1u << ZD));
                const Slot64 *sp[DIM];
#pragma unroll
                for (int dd = 0; dd < DIM; ++dd) sp[dd] = &slot(ch, dd, (vv >> (3 * dd)) & 7);
                M::u3_args(T, f, sp, I.mz[mc][dm - 3][mz_index((vv >> (3 * dm)) & 7, (vv >> (3 * ZD)) & 7)],
                           kk, r200, cc, F);
                out = &I.u3[ch][f][j];
            }
            *out = u_nfw64_F(kk, r200, cc, F);
        }
    }
    __syncthreads();
    for (int p = rank; p < nchild * NP; p += 128) {
        const int ch = p >= NP ? 1 : 0;
        const int pp = p - ch * NP;
        const uint32_t vv = tb.sdesc[pp];
        const Slot64 *sp[DIM];
#pragma unroll
        for (int dd = 0; dd < DIM; ++dd) sp[dd] = &slot(ch, dd, (vv >> (3 * dd)) & 7);
        double uc[NF], u3c[NU3], ax[NA];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            const uint32_t dims = (1u << ucache_fun(KIND, TERM, f, 0)) |
                                  (1u << ucache_fun(KIND, TERM, f, 1)) | (1u << ZD);
            uc[f] = I.uc[ch && own(dims)][f][tb.ucidx[f * NP + pp]];
        }
#pragma unroll
        for (int f = 0; f < NU3; ++f)
            u3c[f] = I.u3[ch && own(7u | (1u << u3_mass(KIND, TERM, f)) | (1u << ZD))][f]
                         [tb.u3rep[f * NP + pp]];
#pragma unroll
        for (int a = 0; a < NA; ++a)
            ax[a] = I.aux[ch && own(aux_dims(TERM, a))][aux_off(TERM, a) + tb.auxrep[a * NP + pp]];
        const double v = M::point(T, d, sp, uc, u3c, ax);
        I.vals[p] = v;
        if (dbg) dbg[p] = v;
    }
    __syncthreads();
    if (rank < 32) {
        double val, err;
        int split;
        const int ch = (lane >> 3) & 1;
        combine64_warp<DIM>(I.vals + (ch < nchild ? ch : 0) * NP, ldexp(d.rootvol, -levsum), val, err,
                            split);
        if ((lane & 7) == 0 && lane < 8 * nchild) {
            const long long slot = lane == 0 ? pslot : qslot;
            P.val[slot] = val;
            P.err[slot] = err;
            P.split[slot] = (unsigned char)split;
            if (P.unc) P.unc[slot] = 0.f;
            if (P.uval) P.uval[slot] = 0.f;
        }
        if (cut && lane < DIM) {
            const int lnew = lane == sdim ? levs : lev;
            P.center[lane * stride + pslot] = lane == sdim ? cL : c_l;
            P.level[lane * stride + pslot] = (unsigned char)lnew;
            P.center[lane * stride + qslot] = lane == sdim ? cR : c_l;
            P.level[lane * stride + qslot] = (unsigned char)lnew;
        }
    }
    __syncthreads();
}

// A block per work item.  (Measured against a warp per item, four per block, which has fewer
// idle lanes at the ends of the passes but leaves a round of few cuts as long as one warp's
// evaluation of a whole cut and an SM's quarters unevenly loaded: the block is as fast or
// faster for rounds of any size, 9 triplets x 3 NMapMap terms 16.0 -> 14.9 ms.)
template <int KIND, int TERM>
__global__ void __launch_bounds__(128, 5) k_eval64(DevTables T, const IntDesc *__restrict__ D,
                                                IntState *__restrict__ S, Pool P, BatchHdr *H,
                                                const long long *__restrict__ woff)
{
    using RT = ReTab<KIND, TERM>;
    __shared__ __align__(16) unsigned char tbuf[sizeof(RT)];
    __shared__ Item64<KIND, TERM> I;
    const int g = KIND * 3 + TERM - 1;
    const int gb = H->gbeg[g], ge = H->gbeg[g + 1];
    if (gb >= ge) return;
    const long long wbeg = woff[gb], wend = woff[ge];
    if (wbeg + blockIdx.x >= wend) return;  // no work here: skip the tables
    const RT &tb = load_retab<KIND, TERM>(P, tbuf);
    for (long long w = wbeg + blockIdx.x; w < wend; w += gridDim.x) {
        int lo = gb, hi = ge - 1;  // last integral i with woff[i] <= w
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (woff[mid] <= w) lo = mid;
            else hi = mid - 1;
        }
        const int i = lo;
        const long long j = w - woff[i];
        const IntDesc &d = D[i];
        const int cj = P.cand[d.base + j];
        const bool cut = cj >= 0;  // cj < 0: a fresh integral's root region
        const long long pslot = d.base + (cut ? cj : 0);
        const long long qslot = cut ? d.base + (S[i].nR - S[i].K) + j : -1;
        // a block's first warps get the passes' uneven remainders: the warp that comes first
        // turns with the item, so that the SM's quarters share them
        const int turn = 32 * (int)((w + (w >> 3) + (w >> 7)) & 3);
        block_item64<KIND, TERM>(T, d, P, pslot, qslot, cut, I, tb, (threadIdx.x + turn) & 127,
                                 &H->ties, H->dbg);
    }
}

static_assert(sizeof(Slot64) == reeval_slot_bytes, "re-evaluation scratch layout");

// FP64 re-evaluation of the regions the mixed-precision pass queued for one group; each
// entry is (integral, local slot | kind << 30): kind 0 = split decision only (the centre
// and the 4 dim axis points enter the fourth differences, src/hcubature.cpp:527-575),
// kind 1 = whole rule (value, error and split: ambiguous selection boundaries and the
// final polish).  The FP64 pipe issues one warp instruction per 64 cycles per SM
// sub-partition, so a round's re-evaluation time is set by the busiest sub-partition and, in
// a round of few entries, by the longest chain of one thread: the work is spread evenly over
// the whole device in three passes over the first P.rcap entries.
//   k_re_fill    coordinate slots; a mass's two populations, its r_200 and its NFW
//                normalisations on threads of their own
//   k_re_ucache  shared u_NFW, two threads each (Si and Ci of either argument), and the
//                auxiliary functions
//   k_re_finish  a block per entry: the points, then the sums in the reference's order
// Every pass's kinds of task start on a warp boundary, so that a warp runs one kind.
// Entries beyond P.rcap take the batched kernel k_reeval64.
template <int KIND, int TERM>
struct Reeval {
    static constexpr int DIM = TERM + 4;
    static constexpr int NP = rule_points(DIM);
    static constexpr int NAX = 1 + 4 * DIM;
    static constexpr int NS = DIM * NVAR;
    static constexpr int G = KIND * 3 + TERM - 1;
    __device__ static Slot64 *slots(const Pool &P)
    {
        return (Slot64 *)(P.rscr + (long long)G * P.rscr_group);
    }
    __device__ static double *ucv(const Pool &P)  // [rcap][UC_NF_MAX][UC_MAX]
    {
        return (double *)(P.rscr + (long long)G * P.rscr_group +
                          ((long long)P.rcap * MAX_DIM * NVAR * reeval_slot_bytes + 255) / 256 * 256);
    }
    __device__ static double *u3v(const Pool &P)  // [rcap][U3_NF_MAX][U3_MAX]
    {
        return ucv(P) + (long long)P.rcap * UC_NF_MAX * UC_MAX;
    }
    __device__ static double *auxv(const Pool &P)  // [rcap][AUX_MAX]
    {
        return u3v(P) + (long long)P.rcap * U3_NF_MAX * U3_MAX;
    }
    __device__ static double *mzv(const Pool &P)  // [rcap][3][MZ_PAIRS][MZ_VALS]
    {
        return auxv(P) + (long long)P.rcap * AUX_MAX;
    }
    __device__ static int ulist_cap(const Pool &P)
    {
        return P.rcap * (NCU + NCU3);
    }
    __device__ static uint32_t *ulist(const Pool &P)  // the stage's u_NFW tasks
    {
        return (uint32_t *)(mzv(P) + (long long)P.rcap * 3 * MZ_PAIRS * MZ_VALS);
    }
    __device__ static double *mz(const Pool &P, int k, int mdim, uint32_t vv)
    {
        const int vm = (vv >> (3 * mdim)) & 7, vz = (vv >> (3 * (DIM - 1))) & 7;
        return mzv(P) + (((long long)k * 3 + (mdim - 3)) * MZ_PAIRS + mz_index(vm, vz)) * MZ_VALS;
    }
    // auxiliary values per entry (124 for the 2-halo terms)
    static constexpr int NAUX = aux_off(TERM, aux_nfun(TERM) - 1) + aux_count(TERM, aux_nfun(TERM) - 1);
    static_assert(NAUX <= AUX_MAX, "auxiliary projections exceed AUX_MAX");
    __device__ static int count(const Pool &P, const BatchHdr *H, int stage)
    {
        const int cap = H->esc_cap[G];
        const int n = H->n_esc[stage][G] < cap ? H->n_esc[stage][G] : cap;
        return n < P.rcap ? n : P.rcap;
    }
    // u_NFW tasks of m entries: [0, m NCU) the (l, m, z) combinations, then the k3 projections
    static constexpr int NCU = ucache_nf(TERM) * UC_MAX, NCU3 = u3_nfun(TERM) * U3_MAX;
    // are they listed first (ULIST_MIN)?
    __device__ static bool u_listed(const Pool &P, int m) { return m * (NCU + NCU3) > P.ulist_min; }
    // does the entry need combination j of function f (split only: those of the centre and one
    // contender axis), and the k3 projection pr?
    __device__ static bool need_uc(const Pool &P, const IntDesc &d, int2 ent, const ReTab<KIND, TERM> &tb,
                                   int f, int j)
    {
        if (j >= tb.ucn[f]) return false;
        if (ent.y >> 30) return true;
        const uint32_t key = tb.ucl[f * UC_MAX + j];
        const int vl = key & 7, vm = (key >> 3) & 7, vz = (key >> 6) & 7;
        const unsigned cm = split_cmask(P, d, ent);
        return (vl != 0) + (vm != 0) + (vz != 0) <= 1 &&
               split_variant(cm, ucache_fun(KIND, TERM, f, 0), vl) &&
               split_variant(cm, ucache_fun(KIND, TERM, f, 1), vm) && split_variant(cm, DIM - 1, vz);
    }
    __device__ static bool need_u3(const Pool &P, const IntDesc &d, int2 ent, int pr)
    {
        return (ent.y >> 30) || split_point(split_cmask(P, d, ent), pr, NAX);
    }
    // coordinate of variant v of dimension dim of entry ent
    __device__ static double coord(const Pool &P, const IntDesc &d, int2 ent, int dim, int v)
    {
        const long long slot = d.base + (ent.y & 0x3FFFFFFF);
        return variant_x(P.center[dim * P.stride + slot],
                         ldexp(d.hw0[dim], -(int)P.level[dim * P.stride + slot]), v);
    }
};

__host__ __device__ constexpr long long warps_up(long long n) { return (n + 31) / 32 * 32; }

// The u_NFW tasks are numbered over all entries alike, but a split-only entry needs a few of
// them, and the FP64 pipe takes a warp's instruction in the same time for one lane as for 32
// (11 of 32 were active in k_re_ucache, the largest of the passes).  So k_re_fill lists the
// needed ones, packed over the whole queue, while its other blocks fill the slots: 220
// triplets: 21 of 32 lanes, re-evaluations 22.5 -> 19.2 ms, call 49.1 -> 46.3 ms; 13 triplets
// of two populations 5.3 -> 5.1 ms.  (A block listing its own share only leaves the device
// uneven: 20.0-22.2 ms.  The same for the fill's own tasks gains nothing.)
constexpr int RE_CHUNK = 1024;
struct ReChunk {
    int n, at;
    uint16_t list[RE_CHUNK];
};
// chunk of a pass over `tasks` tasks by the whole grid, in units of a block's threads
__device__ __forceinline__ int re_chunk_size(int tasks, int unit)
{
    const int c = tasks / (int)gridDim.x / unit * unit;
    return c < unit ? unit : (c > RE_CHUNK ? RE_CHUNK : c);
}
// lists the needed tasks of [t0, t0 + size): their count
template <class Need>
__device__ __forceinline__ int re_gather(ReChunk &ck, int t0, int size, const Need &need)
{
    __syncthreads();
    if (threadIdx.x == 0) ck.n = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int i0 = threadIdx.x - lane; i0 < size; i0 += blockDim.x) {
        const int i = i0 + lane;
        const bool on = i < size && need(t0 + i);
        const unsigned b = __ballot_sync(0xffffffffu, on);
        int at = 0;
        if (lane == 0 && b) at = atomicAdd(&ck.n, __popc(b));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (on) ck.list[at + __popc(b & ((1u << lane) - 1u))] = (uint16_t)i;
    }
    __syncthreads();
    return ck.n;
}

template <int KIND, int TERM>
__global__ void __launch_bounds__(128) k_re_fill(DevTables T, const IntDesc *__restrict__ D,
                                                 IntState *__restrict__ S, Pool P, BatchHdr *H,
                                                 const long long *__restrict__ woff, int stage)
{
    using R = Reeval<KIND, TERM>;
    using M = Model64<KIND, TERM>;
    __shared__ ReChunk ck;
    // the second stage's queue of the previous round has been consumed
    if (stage == 0 && blockIdx.x == 0 && threadIdx.x == 0) H->n_esc[1][R::G] = 0;
    const int m = R::count(P, H, stage);
    if (m == 0) return;
    const int2 *Q = P.esc + H->esc_beg[R::G];
    Slot64 *SL = R::slots(P);
    constexpr int ZD = R::DIM - 1, NMS = TERM * NVAR, NLS = 4 * NVAR, NMZ = TERM * MZ_PAIRS;
    // masses (the longest), the second population's occupations, r_200, the normalisations,
    // then l1, l2, phi and z
    const long long b1 = warps_up((long long)m * NMS), b2 = b1 + (KIND == 0 ? b1 : 0);
    const long long nmz = warps_up((long long)m * NMZ), b3 = b2 + nmz, b4 = b3 + nmz;
    const long long tot = b4 + (long long)m * NLS;
    // The u_NFW tasks of k_re_ucache, packed over the whole queue: listed by the other end of
    // the grid, which has no task here in a round of few entries.
    const int nu = R::u_listed(P, m) ? m * (R::NCU + R::NCU3) : 0;
    const int usize = re_chunk_size(nu, 128);
    const int ufirst = (int)(gridDim.x - 1 - blockIdx.x) * usize;
    if (ufirst < nu) {
        const ReTab<KIND, TERM> &tb =
            *reinterpret_cast<const ReTab<KIND, TERM> *>(P.retab + R::G * RETAB_BYTES);
        const auto need_u = [&](int t) {
            const bool uc = t < m * R::NCU;
            const int per = uc ? R::NCU : R::NCU3, t2 = uc ? t : t - m * R::NCU;
            const int k = t2 / per, r = t2 - k * per;
            if (k >= m) return false;
            const int2 ent = Q[k];
            return uc ? R::need_uc(P, D[ent.x], ent, tb, r / UC_MAX, r % UC_MAX)
                      : R::need_u3(P, D[ent.x], ent, tb.u3list[r]);
        };
        uint32_t *U = R::ulist(P);
        for (int t0 = ufirst; t0 < nu; t0 += (int)gridDim.x * usize) {
            const int n = re_gather(ck, t0, usize, need_u);
            if (threadIdx.x == 0) ck.at = atomicAdd(&H->n_ulist[R::G], n);
            __syncthreads();
            for (int u = threadIdx.x; u < n; u += blockDim.x)
                if (ck.at + u < R::ulist_cap(P)) U[ck.at + u] = (uint32_t)(t0 + ck.list[u]);
        }
    }
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < tot;
         t += (long long)gridDim.x * blockDim.x) {
        if (t < b2) {
            const bool second = t >= b1;
            const long long q = second ? t - b1 : t;
            const int k = (int)(q / NMS), r = (int)(q - (long long)k * NMS);
            if (k >= m) continue;
            const int dim = 3 + r / NVAR, v = r % NVAR;
            const int2 ent = Q[k];
            const IntDesc &d = D[ent.x];
            if (second && d.same) continue;
            // split only: the centre of every dimension, the contenders' axis variants
            if (!(ent.y >> 30) && !split_variant(split_cmask(P, d, ent), dim, v)) continue;
            const double x = R::coord(P, d, ent, dim, v);
            Slot64 &sl = SL[(long long)k * R::NS + dim * NVAR + v];
            if (!second) {
                Slot64 f;
                M::fill_mass(T, d, x, f, &H->ties);
                sl.a[0] = f.a[0];
                sl.a[1] = f.a[1];
                sl.a[2] = f.a[2];
                sl.i0 = f.i0;
                sl.i1 = f.i1;
                if (KIND == 0 && d.same) {
                    sl.a[3] = f.a[3];
                    sl.a[4] = f.a[4];
                    sl.a[5] = f.a[5];
                }
            } else {
                occupations64(T.hod + 6 * d.hod2, pow(10, x), sl.a[3], sl.a[4]);
            }
        } else if (t < b4) {
            // r_200 and F of the (mass, z) pairs, from the mass slot's expressions
            const bool norm = t >= b3;
            const long long q = t - (norm ? b3 : b2);
            const int k = (int)(q / NMZ), r = (int)(q - (long long)k * NMZ);
            if (k >= m) continue;
            const int md = 3 + r / MZ_PAIRS, j = r - (md - 3) * MZ_PAIRS;
            const int vm = mz_vm_of(j), vz = mz_vz_of(j);
            const int2 ent = Q[k];
            const IntDesc &d = D[ent.x];
            if (!(ent.y >> 30)) {
                const unsigned cm = split_cmask(P, d, ent);
                if ((vm && vz) || !split_variant(cm, md, vm) || !split_variant(cm, ZD, vz)) continue;
            }
            const double xm = R::coord(P, d, ent, md, vm);
            const int zt = z_trunc64(T, R::coord(P, d, ent, ZD, vz));
            double *o = R::mzv(P) + (((long long)k * 3 + (md - 3)) * MZ_PAIRS + j) * MZ_VALS;
            if (norm) {
                Slot64 f;
                m_index_x(T, xm, f.i0, f.i1);
                M::mz_norms(T, d, f, zt, KIND == 0 ? 3 : 2, o);
            } else {
                o[0] = r200_64(pow(10, xm), __ldg(T.rho_bar + zt));
            }
        } else {
            const long long q = t - b4;
            const int k = (int)(q / NLS), r = (int)(q - (long long)k * NLS);
            const int dim = r / NVAR < 3 ? r / NVAR : ZD, v = r % NVAR;
            const int2 ent = Q[k];
            const IntDesc &d = D[ent.x];
            if (!(ent.y >> 30) && !split_variant(split_cmask(P, d, ent), dim, v)) continue;
            M::fill(T, d, dim, R::coord(P, d, ent, dim, v), SL[(long long)k * R::NS + dim * NVAR + v],
                    &H->ties);
        }
    }
}

// u_NFW of each entry's (l, m, z) combinations and k3 projections (whole rules: all of them;
// split only: those that the centre and the contenders' axis points read), then the
// auxiliary functions per projection and the satellite pair counts of two populations.
template <int KIND, int TERM>
__global__ void __launch_bounds__(128) k_re_ucache(DevTables T, const IntDesc *__restrict__ D,
                                                   IntState *__restrict__ S, Pool P, BatchHdr *H,
                                                   const long long *__restrict__ woff, int stage)
{
    using R = Reeval<KIND, TERM>;
    using M = Model64<KIND, TERM>;
    constexpr int NF = ucache_nf(TERM), NU3 = u3_nfun(TERM), ZD = R::DIM - 1;
    __shared__ __align__(16) unsigned char tbuf[sizeof(ReTab<KIND, TERM>)];
    __shared__ double ex[3][64];
    const int m = R::count(P, H, stage);
    if (m == 0) return;
    const int b1 = m * R::NCU;
    const bool listed = R::u_listed(P, m);
    const int nu = listed ? min(H->n_ulist[R::G], R::ulist_cap(P)) : m * (R::NCU + R::NCU3);
    const long long a1 = warps_up((long long)m * R::NAUX);
    const long long na = a1 + (KIND == 0 ? (long long)m * TERM * NVAR : 0);
    // the auxiliary tasks start from the other end of the grid
    const long long first_aux = (long long)(gridDim.x - 1 - blockIdx.x) * blockDim.x;
    if ((int)blockIdx.x * 64 >= nu && first_aux >= na) return;  // no work here: skip the tables
    const ReTab<KIND, TERM> &tb = load_retab<KIND, TERM>(P, tbuf);
    const int2 *Q = P.esc + H->esc_beg[R::G];
    Slot64 *SL = R::slots(P);
    double *UC = R::ucv(P), *U3C = R::u3v(P), *AX = R::auxv(P);
    const int part = threadIdx.x >> 6, q = threadIdx.x & 63;
    const uint32_t *U = R::ulist(P);
    const int tend = b1 + m * R::NCU3;
    for (int u0 = (int)blockIdx.x * 64; u0 < nu; u0 += (int)gridDim.x * 64) {
        double kk = 1, r200 = 1, cc = 1, F = 1;
        double *out = nullptr;
        const int t = u0 + q < nu ? (listed ? (int)U[u0 + q] : u0 + q) : tend;
        if (t < b1) {
            const int k = t / R::NCU, r = t - k * R::NCU;
            const int f = r / UC_MAX, j = r - f * UC_MAX;
            const int2 ent = Q[k];
            const IntDesc &d = D[ent.x];
            if (listed || R::need_uc(P, d, ent, tb, f, j)) {
                const uint32_t key = tb.ucl[f * UC_MAX + j];
                const int vl = key & 7, vm = (key >> 3) & 7, vz = (key >> 6) & 7;
                const int dl = ucache_fun(KIND, TERM, f, 0), dm = ucache_fun(KIND, TERM, f, 1);
                const Slot64 *base = SL + (long long)k * R::NS;
                M::ucached_args(T, d, f, base[dl * NVAR + vl], base[dm * NVAR + vm], base[ZD * NVAR + vz],
                                R::mz(P, k, dm, ((uint32_t)vm << (3 * dm)) | ((uint32_t)vz << (3 * ZD))),
                                kk, r200, cc, F);
                out = UC + ((long long)k * UC_NF_MAX + f) * UC_MAX + j;
            }
        } else if (t < tend) {
            const int t2 = t - b1;
            const int k = t2 / R::NCU3, r = t2 - k * R::NCU3;
            const int2 ent = Q[k];
            const int pr = tb.u3list[r];  // every projection index is used (93)
            if (listed || R::need_u3(P, D[ent.x], ent, pr)) {
                const int f = r / U3_MAX, j = r - f * U3_MAX;
                const uint32_t vv = tb.sdesc[pr];
                const Slot64 *base = SL + (long long)k * R::NS;
                const Slot64 *sp[R::DIM];
#pragma unroll
                for (int dd = 0; dd < R::DIM; ++dd) sp[dd] = base + dd * NVAR + ((vv >> (3 * dd)) & 7);
                M::u3_args(T, f, sp, R::mz(P, k, u3_mass(KIND, TERM, f), vv), kk, r200, cc, F);
                out = U3C + ((long long)k * U3_NF_MAX + f) * U3_MAX + j;
            }
        }
        // u_nfw64_F, each argument's Si and Ci on a thread of its own (64 apart)
        const double arg1 = ddiv(kk * r200, cc);
        const double arg2 = arg1 * (1 + cc);
        double si = 0, ci = 0, sx = 0, cx = 0;
        if (out) sici64_sc(part ? arg2 : arg1, si, ci, sx, cx);
        if (part) {
            ex[0][q] = si;
            ex[1][q] = ci;
            if (out) ex[2][q] = ddiv(-sin(arg1 * cc), arg2);
        }
        __syncthreads();
        if (!part && out) {
            const double term1 = sx * (ex[0][q] - si);
            const double term2 = cx * (ex[1][q] - ci);
            *out = ddiv(term1 + term2 + ex[2][q], F);
        }
        __syncthreads();
    }
    for (long long t = first_aux + threadIdx.x; t < na; t += (long long)gridDim.x * blockDim.x) {
        if (t >= a1) {
            const long long t2 = t - a1;
            const int k = (int)(t2 / (TERM * NVAR)), r = (int)(t2 - (long long)k * (TERM * NVAR));
            const int2 ent = Q[k];
            const IntDesc &d = D[ent.x];
            if (d.same || (!(ent.y >> 30) && !split_variant(split_cmask(P, d, ent), 3 + r / NVAR, r % NVAR)))
                continue;
            Slot64 &sl = SL[(long long)k * R::NS + 3 * NVAR + r];
            sl.a[5] = M::pairs(T, d, sl);
            continue;
        }
        const int k = (int)(t / R::NAUX), r = (int)(t - (long long)k * R::NAUX);
        if (k >= m) continue;
        int a = 0;
        while (a + 1 < aux_nfun(TERM) && r >= aux_off(TERM, a + 1)) ++a;
        const int pr = tb.auxlist[r];
        const int2 ent = Q[k];
        // split only: the projections of the centre and the contenders' axis points
        if (!(ent.y >> 30) && !split_point(split_cmask(P, D[ent.x], ent), pr, R::NAX)) continue;
        const uint32_t vv = tb.sdesc[pr];
        const Slot64 *base = SL + (long long)k * R::NS;
        const Slot64 *sp[R::DIM];
#pragma unroll
        for (int dd = 0; dd < R::DIM; ++dd) sp[dd] = base + dd * NVAR + ((vv >> (3 * dd)) & 7);
        AX[(long long)k * AUX_MAX + r] = M::aux(T, D[ent.x], a, sp);
    }
}

// the split dimension of one re-taken split (vl: its rule-point values; cm: the contenders)
template <int DIM>
__device__ int retaken_split(const double *vl, unsigned cm)
{
    const double ratio = (G3L_LAMBDA2 * G3L_LAMBDA2) / (G3L_LAMBDA4 * G3L_LAMBDA4);
    const double val0 = vl[0];
    double maxdiff = 0;
    int dimDiffMax = 0;
    for (int q = 0; q < DIM; ++q) {
        if (!((cm >> q) & 1u)) continue;  // not a contender (its points were not taken)
        double v0 = vl[1 + 4 * q], v1 = vl[2 + 4 * q];
        double v2 = vl[3 + 4 * q], v3 = vl[4 + 4 * q];
        double diff = 0;
        diff += fabs(v0 + v1 - 2 * val0 - ratio * (v2 + v3 - 2 * val0));
        if (diff > maxdiff) {
            maxdiff = diff;
            dimDiffMax = q;
        }
    }
    return dimDiffMax;
}

// the sums of one re-evaluated region by one warp (vl: its rule-point values)
template <int DIM>
__device__ void reeval_finish(const IntDesc &d, const Pool &P, long long slot, bool full,
                              const double *vl, unsigned cm)
{
    const int lane = threadIdx.x & 31;
    if (full) {
        const int lsum = __reduce_add_sync(0xffffffffu, lane < DIM ? (int)P.level[lane * P.stride + slot] : 0);
        double val, err;
        int split;
        combine64_warp<DIM>(vl, ldexp(d.rootvol, -lsum), val, err, split);
        if (lane == 0) {
            P.val[slot] = val;
            P.err[slot] = err;
            P.split[slot] = (unsigned char)split;
            P.unc[slot] = 0.f;
            P.uval[slot] = 0.f;
        }
    } else if (lane == 0) {
        P.split[slot] = (unsigned char)retaken_split<DIM>(vl, cm);
    }
}

template <int KIND, int TERM>
__global__ void __launch_bounds__(128) k_re_finish(DevTables T, const IntDesc *__restrict__ D,
                                                   IntState *__restrict__ S, Pool P, BatchHdr *H,
                                                   const long long *__restrict__ woff, int stage)
{
    using R = Reeval<KIND, TERM>;
    constexpr int DIM = R::DIM, NF = ucache_nf(TERM), NU3 = u3_nfun(TERM), NA = aux_nfun(TERM);
    __shared__ __align__(16) unsigned char tbuf[sizeof(ReTab<KIND, TERM>)];
    __shared__ double vals[R::NP];
    const int m = R::count(P, H, stage);
    if (blockIdx.x == 0 && threadIdx.x == 0) H->n_ulist[R::G] = 0;  // consumed by k_re_ucache
    if ((int)blockIdx.x >= m) return;  // no work here: skip the tables
    const ReTab<KIND, TERM> &tb = load_retab<KIND, TERM>(P, tbuf);
    const int2 *Q = P.esc + H->esc_beg[R::G];
    const Slot64 *SL = R::slots(P);
    const double *UC = R::ucv(P), *U3C = R::u3v(P), *AX = R::auxv(P);
    for (int k = blockIdx.x; k < m; k += gridDim.x) {
        const int2 ent = Q[k];
        const IntDesc &d = D[ent.x];
        const bool full = (ent.y >> 30) != 0;
        const unsigned cm = full ? 0u : split_cmask(P, d, ent);
        for (int p = threadIdx.x; p < (full ? R::NP : R::NAX); p += 128) {
            if (!full && !split_point(cm, p, R::NAX)) continue;
            const uint32_t vv = tb.sdesc[p];
            const Slot64 *base = SL + (long long)k * R::NS;
            const Slot64 *sp[DIM];
#pragma unroll
            for (int dd = 0; dd < DIM; ++dd) sp[dd] = base + dd * NVAR + ((vv >> (3 * dd)) & 7);
            double uc[NF], u3c[NU3], ax[NA];
#pragma unroll
            for (int f = 0; f < NF; ++f)
                uc[f] = UC[((long long)k * UC_NF_MAX + f) * UC_MAX + tb.ucidx[f * R::NP + p]];
#pragma unroll
            for (int f = 0; f < NU3; ++f)
                u3c[f] = U3C[((long long)k * U3_NF_MAX + f) * U3_MAX + tb.u3rep[f * R::NP + p]];
#pragma unroll
            for (int a = 0; a < NA; ++a)
                ax[a] = AX[(long long)k * AUX_MAX + aux_off(TERM, a) + tb.auxrep[a * R::NP + p]];
            vals[p] = Model64<KIND, TERM>::point(T, d, sp, uc, u3c, ax);
        }
        __syncthreads();
        if (threadIdx.x < 32)
            reeval_finish<DIM>(d, P, d.base + (ent.y & 0x3FFFFFFF), full, vals, cm);
        __syncthreads();
    }
}

// Entries beyond P.rcap: a block takes a batch of RB entries and spreads their slots and
// points over its threads (shared-memory staging, no scratch).
template <int KIND, int TERM>
__global__ void __launch_bounds__(128) k_reeval64(DevTables T, const IntDesc *__restrict__ D,
                                                  IntState *__restrict__ S, Pool P, BatchHdr *H,
                                                  const long long *__restrict__ woff, int stage)
{
    constexpr int DIM = TERM + 4;
    constexpr int NP = rule_points(DIM);
    constexpr int NAX = 1 + 4 * DIM;
    constexpr int RB = 4;  // entries per batch
    constexpr int NS = DIM * NVAR;
    __shared__ uint32_t sdesc[NP];
    __shared__ Slot64 slots[RB][NS];
    __shared__ double vals[RB][NP];
    __shared__ int2 sent[RB];
    const int g = KIND * 3 + TERM - 1;
    const int cap = H->esc_cap[g];
    const int n = H->n_esc[stage][g] < cap ? H->n_esc[stage][g] : cap;
    const int first = P.rcap;
    if (n <= first) return;
    for (int p = threadIdx.x; p < NP; p += blockDim.x) sdesc[p] = point_variants(DIM, p);
    const int2 *Q = P.esc + H->esc_beg[g];
    const long long stride = P.stride;
    const int nb = (n - first + RB - 1) / RB;
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        const int e0 = first + b * RB;
        const int ne = n - e0 < RB ? n - e0 : RB;
        __syncthreads();
        if (threadIdx.x < ne) sent[threadIdx.x] = Q[e0 + threadIdx.x];
        __syncthreads();
        for (int t = threadIdx.x; t < ne * NS; t += blockDim.x) {
            const int k = t / NS, r = t - k * NS;
            const int dim = r / NVAR, v = r - dim * NVAR;
            const int2 ent = sent[k];
            const IntDesc &d = D[ent.x];
            if (!(ent.y >> 30) && !split_variant(split_cmask(P, d, ent), dim, v)) continue;
            const long long slot = d.base + (ent.y & 0x3FFFFFFF);
            const double c = P.center[dim * stride + slot];
            const double hw = ldexp(d.hw0[dim], -(int)P.level[dim * stride + slot]);
            double x = c;
            if (v > 0) {
                double lam = (v <= 2) ? G3L_LAMBDA2 : (v <= 4 ? G3L_LAMBDA4 : G3L_LAMBDA5);
                double rr = hw * lam;
                x = (v & 1) ? c - rr : c + rr;
            }
            Model64<KIND, TERM>::fill(T, d, dim, x, slots[k][r], &H->ties);
        }
        __syncthreads();
        int pb[RB + 1];
        pb[0] = 0;
#pragma unroll
        for (int k = 0; k < RB; ++k)
            pb[k + 1] = pb[k] + (k < ne ? ((sent[k].y >> 30) ? NP : NAX) : 0);
        for (int t = threadIdx.x; t < pb[RB]; t += blockDim.x) {
            int k = 0;
#pragma unroll
            for (int q = 1; q < RB; ++q) k += t >= pb[q] ? 1 : 0;
            const int p = t - pb[k];
            const IntDesc &d = D[sent[k].x];
            if (!(sent[k].y >> 30) && !split_point(split_cmask(P, d, sent[k]), p, NAX)) continue;
            const uint32_t vv = sdesc[p];
            const Slot64 *sp[DIM];
#pragma unroll
            for (int dd = 0; dd < DIM; ++dd) sp[dd] = &slots[k][dd * NVAR + ((vv >> (3 * dd)) & 7)];
            vals[k][p] = Model64<KIND, TERM>::point(T, d, sp);
        }
        __syncthreads();
        static_assert(RB <= 4, "one warp per entry");
        if ((int)threadIdx.x >> 5 < ne) {
            const int2 ent = sent[threadIdx.x >> 5];
            const IntDesc &d = D[ent.x];
            reeval_finish<DIM>(d, P, d.base + (ent.y & 0x3FFFFFFF), (ent.y >> 30) != 0,
                               vals[threadIdx.x >> 5], (ent.y >> 30) ? 0u : split_cmask(P, d, ent));
        }
    }
}

#define G3L_INST64(K, Tm)                                                                        \
    template __global__ void k_eval64<K, Tm>(DevTables, const IntDesc *, IntState *, Pool,      \
                                             BatchHdr *, const long long *);                     \
    template __global__ void k_reeval64<K, Tm>(DevTables, const IntDesc *, IntState *, Pool,    \
                                               BatchHdr *, const long long *, int);              \
    template __global__ void k_re_fill<K, Tm>(DevTables, const IntDesc *, IntState *, Pool,     \
                                              BatchHdr *, const long long *, int);               \
    template __global__ void k_re_ucache<K, Tm>(DevTables, const IntDesc *, IntState *, Pool,   \
                                                BatchHdr *, const long long *, int);             \
    template __global__ void k_re_finish<K, Tm>(DevTables, const IntDesc *, IntState *, Pool,   \
                                                BatchHdr *, const long long *, int);             \
    template __global__ void k_re_tables<K, Tm>(unsigned char *);
G3L_INST64(0, 1)
G3L_INST64(0, 2)
G3L_INST64(0, 3)
G3L_INST64(1, 1)
G3L_INST64(1, 2)
G3L_INST64(1, 3)

// Build the re-evaluation point tables of every group into out (NGROUPS * RETAB_BYTES
// bytes of device memory), on stream s.
cudaError_t build_reeval_tables(unsigned char *out, cudaStream_t s)
{
    k_re_tables<0, 1><<<1, 128, 0, s>>>(out);
    k_re_tables<0, 2><<<1, 128, 0, s>>>(out);
    k_re_tables<0, 3><<<1, 128, 0, s>>>(out);
    k_re_tables<1, 1><<<1, 128, 0, s>>>(out);
    k_re_tables<1, 2><<<1, 128, 0, s>>>(out);
    k_re_tables<1, 3><<<1, 128, 0, s>>>(out);
    return cudaGetLastError();
}

// re-evaluation kernels of a group: 0 = fill, 1 = cached values, 2 = points and sums,
// 3 = batched tail
void *reeval_phase_kernel(int kind, int term, int phase)
{
#define G3L_RE_ROW(K, Tm)                                                                       \
    {(void *)k_re_fill<K, Tm>, (void *)k_re_ucache<K, Tm>, (void *)k_re_finish<K, Tm>,           \
     (void *)k_reeval64<K, Tm>}
    static void *tab[2][3][4] = {{G3L_RE_ROW(0, 1), G3L_RE_ROW(0, 2), G3L_RE_ROW(0, 3)},
                                 {G3L_RE_ROW(1, 1), G3L_RE_ROW(1, 2), G3L_RE_ROW(1, 3)}};
#undef G3L_RE_ROW
    return tab[kind][term - 1][phase];
}

void *eval64_kernel(int kind, int term)
{
    static void *tab[2][3] = {
        {(void *)k_eval64<0, 1>, (void *)k_eval64<0, 2>, (void *)k_eval64<0, 3>},
        {(void *)k_eval64<1, 1>, (void *)k_eval64<1, 2>, (void *)k_eval64<1, 3>}};
    return tab[kind][term - 1];
}

}  // namespace g3l
