// sm_ecyl.cu -- e_cyl_iso (2.5-D elastic FDTD in cylindrical coordinates r, z
// with azimuthal mode n, CPML) on sm_100a.
//
// Grid.  The reference's padded grid: nx2 = nx + np radial columns (the
// absorbing layer only beyond r = (nx-1) dr; r = 0 is the axis) by
// nz2 = nz + 2 np rows; here each column is padded to `pitch` cells so rows
// start aligned.  Nine fields (vr vt vz trr ttt tzz trz trt ttz) are updated
// in place: one launch updates the three velocities from the stresses
// (e_cyl_iso.c:612-633) and adds the force sources (src.c:186-199), one
// updates the six stresses from the velocities (e_cyl_iso.c:640-662) and adds a
// Kurkjian source (src.c:231-236); the two also sample the receivers
// (ECylServe).  z is the fast index.
// Away from the absorbing layers, the axis and the last column a thread owns
// 16 bytes of consecutive z cells (ECylVec) of one column; everywhere else a
// thread owns one cell (ECylSplit says which cells go where).
//
// Arithmetic.  Each update keeps the reference's expression and order of
// operations (propagate.c:2706-3309 for mode 0, :3312-4088 for n > 0); this
// file is compiled without FMA contraction, so the FP64 build follows the
// FP64 reference to the last bit where the reference is built the same way.
// The FP32 build multiplies by reciprocals of the grid lengths instead of
// dividing (ECylQ); the FP64 vector path forms the correctly rounded quotient
// from the reciprocal (ECylF).
// Materials arrive multiplied by dt on the host in FP64 (the reference's
// dt*b*(...) evaluates dt*b first).
//
// CPML memory variables.  z-side variables live in nx2 x (2 np + 1) strips
// (slot j below the interior, np + j - (nz + np - 1) above it), r-side ones
// in (np + 1) x nz2 strips (slot i - (nx - 1) for half-node updates, i - nx
// for node updates): every cell owns its own variable.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <vector>

#include "sm_common.cuh"

namespace sm {

enum { C_VR, C_VT, C_VZ, C_TRR, C_TTT, C_TZZ, C_TRZ, C_TRT, C_TTZ };
enum { CM_L, CM_L2M, CM_MU, CM_MUI, CM_MUJ, CM_BI, CM_BJ, CM_BIJ };
// coefficient arrays (np each, then np + 1 each)
enum { K_IKR, K_IKZ, K_IKHZ, K_BR, K_CR, K_BZ, K_CZ, K_BHZ, K_CHZ,
       K_IKHR_E, K_IKHZ_E, K_BHR_E, K_CHR_E, K_BHZ_E, K_CHZ_E };
enum { ZV_TRZ, ZV_TTZ, ZV_TZZ, ZV_VZ, ZV_VR, ZV_VT, NZV };
enum { RV_DTRR, RV_TRR1, RV_TRT1, RV_TTT1, RV_TRT2, RV_DTRT, RV_TTT2, RV_DTRZ, RV_TRZ, RV_TTZ,
       RV_DVR, RV_VR1, RV_VT1, RV_DVZ, RV_DVT, RV_VR2, RV_VT2, RV_VZ, NRV };

template <typename C>
struct ECylArgs {
    int nx, nz, np, nx2, nz2, pitch, n;
    C dx, dz, idx, idz;   // and 1/dx, 1/dz
    // per column 1/(2 i dx), 1/(i dx), 1/((i+1/2) dx), 1/(2 (i+1/2) dx).  In FP64 these and
    // idx, idz have to be the correctly rounded reciprocals of exactly the
    // lengths that ECylF forms: its quotients rest on that.
    const C *inv;
    C *f[9];
    const C *m[8];    // dt * (lij l2mij mu mui muj bi bj bij)
    const C *k;       // the 15 coefficient arrays, back to back
    C *zm;            // NZV strips of nx2 * (2 np + 1)
    C *rm;            // NRV strips of (np + 1) * nz2
};

// Which cells the two launches update with 16-byte vectors: columns
// [1, nx - 2] and rows [ja, jb), jb - ja a multiple of the vector; the cells
// around them (the axis column, the columns from nx - 1 on, the rows below ja
// and from jb on) go one to a thread.  The single-cell CTAs come first in the
// grid: they are few and take longer, so they start before the vector CTAs
// fill the device.
struct ECylSplit {
    int ja, jb;      // vector rows (ja == jb: none, every cell on its own)
    int nlane;       // (jb - ja) / cells per vector
    int nvb;         // vector CTAs per column
    int nsingle;     // CTAs of single cells
    int nfull;       // cells of the columns taken whole
};
constexpr int kECylThreads = 128;

template <typename C>
struct ECylDev {
    const ECylArgs<C> &a;
    int i, j;
    __device__ C F(int k, int ii, int jj) const { return a.f[k][(long long)ii * a.pitch + jj]; }
    // a field this launch only reads (not through the read-only path: the launch
    // before may still be writing it when this one starts, see chain_wait)
    __device__ C G(int k, int ii, int jj) const { return F(k, ii, jj); }
    __device__ C M(int k) const { return __ldg(a.m[k] + (long long)i * a.pitch + j); }
    __device__ C K(int arr, int idx) const {
        const int np = a.np;
        const int off = arr < 9 ? arr * np : 9 * np + (arr - 9) * (np + 1);
        return a.k[off + idx];
    }
    // one row below, as the reference's flat index reads it: with no PML the
    // row -1 of column i is row nz2-1 of column i-1, and before the array
    // (i = 0) it is taken as zero
    __device__ C below(int k) const {
        if (j > 0) return G(k, i, j - 1);
        return i > 0 ? G(k, i - 1, a.nz2 - 1) : C(0);
    }
    __device__ C cpml(C *psi, C b, C c, C ik, C d) const {
        const C p = b * *psi + c * d;
        *psi = p;
        return ik * d + p;
    }
    __device__ C *zvar(int v) const {
        const int np = a.np;
        const int s = j < np ? j : np + (j - (a.nz + np - 1));
        return a.zm + ((long long)v * a.nx2 + i) * (2 * np + 1) + s;
    }
    __device__ C *rvar(int v, int slot) const {
        return a.rm + ((long long)v * (a.np + 1) + slot) * a.nz2 + j;
    }
    __device__ bool zhalf() const { return j < a.np || j >= a.nz + a.np - 1; }
    __device__ bool znode() const { return j < a.np || j >= a.nz + a.np; }
    // z filters: h/H coefficients (vr, vt, taa), node coefficients mirrored
    // above (vz, ttz), h/H with rows from 1 (trz)
    __device__ C zf_half(int v, C d) const {
        const int top = a.nz + a.np - 1;
        if (j < a.np) return cpml(zvar(v), K(K_BHZ, j), K(K_CHZ, j), K(K_IKHZ, j), d);
        const int jj = j - top;
        return cpml(zvar(v), K(K_BHZ_E, jj), K(K_CHZ_E, jj), K(K_IKHZ_E, jj), d);
    }
    __device__ C zf_node(int v, C d) const {
        const int top = a.nz + a.np;
        if (j < a.np) return cpml(zvar(v), K(K_BZ, j), K(K_CZ, j), K(K_IKZ, j), d);
        const int q = a.np - 1 - (j - top);
        return cpml(zvar(v), K(K_BZ, q), K(K_CZ, q), K(K_IKZ, q), d);
    }
    __device__ C zf_trz(C d) const {
        const int top = a.nz + a.np;
        if (j < a.np) return cpml(zvar(ZV_VR), K(K_BHZ, j), K(K_CHZ, j), K(K_IKHZ, j), d);
        const int jj = j - top;
        return cpml(zvar(ZV_VR), K(K_BHZ_E, jj), K(K_CHZ_E, jj), K(K_IKHZ_E, jj), d);
    }
    // r filters beyond the interior: node (i >= nx, mirrored node
    // coefficients) and half node (i >= nx-1, the H coefficients)
    __device__ C rf_node(int v, C d) const {
        const int ii = i - a.nx, q = a.np - 1 - ii;
        return cpml(rvar(v, ii), K(K_BR, q), K(K_CR, q), K(K_IKR, q), d);
    }
    __device__ C rf_half(int v, C d) const {
        const int ii = i - (a.nx - 1);
        return cpml(rvar(v, ii), K(K_BHR_E, ii), K(K_CHR_E, ii), K(K_IKHR_E, ii), d);
    }
};

// Quotients by the grid's lengths: dx, dz, 2 i dx, i dx, (i + 1/2) dx and
// 2 (i + 1/2) dx.  FP64 divides, as the reference does; FP32 multiplies by
// reciprocals formed in FP64 on the host (per column), which keeps the FP32
// path far from its own error bound and avoids the division routine.
template <typename C>
struct ECylQ {
    static constexpr bool exact = sizeof(C) == 8;
    C dx, dz, idx, idz;
    C r2i, ri, r5, r25;       // denominators of column i (exact path)
    C i2i, ii, i5, i25;       // their reciprocals (FP32 path)
    __device__ ECylQ(const ECylArgs<C> &a, int i) : dx(a.dx), dz(a.dz), idx(a.idx), idz(a.idz) {
        r2i = C(2.) * C(i) * dx;
        ri = C(i) * dx;
        r5 = (C(i) + C(0.5)) * dx;
        r25 = C(2.) * (C(i) + C(0.5)) * dx;
        if (!exact) {
            const long long s = a.nx2;
            i2i = a.inv[i];
            ii = a.inv[s + i];
            i5 = a.inv[2 * s + i];
            i25 = a.inv[3 * s + i];
        }
    }
    __device__ C x(C v) const { return exact ? v / dx : v * idx; }
    __device__ C z(C v) const { return exact ? v / dz : v * idz; }
    __device__ C twoi(C v) const { return exact ? v / r2i : v * i2i; }
    __device__ C i1(C v) const { return exact ? v / ri : v * ii; }
    __device__ C half(C v) const { return exact ? v / r5 : v * i5; }
    __device__ C twohalf(C v) const { return exact ? v / r25 : v * i25; }
};

// The same quotients for the vector path.  FP32: ECylQ's products.  FP64: the
// correctly rounded quotient without a division, from the correctly rounded
// reciprocal r of the denominator (Markstein, IBM J. Res. Dev. 34, 1990): two
// corrections q += (v - q d) r of q = v r; the first leaves q within one ulp,
// so the second remainder is exact and its rounding is that of v / d.  That
// holds while nothing under- or overflows: `ok` turns false when a numerator
// is not zero and not in [2^-960, 2^900) (the remainder's last bit is 2^-104 of
// it; infinities and NaN included), and the caller then divides.  A division costs about 25
// instructions with its range tests; this is 5 and the test 3.
template <typename C>
struct ECylF : ECylQ<C> {
    bool ok = true;
    __device__ ECylF(const ECylArgs<C> &a, int i) : ECylQ<C>(a, i) {}
    __device__ C x(C v) { return this->ECylQ<C>::x(v); }
    __device__ C z(C v) { return this->ECylQ<C>::z(v); }
    __device__ C twoi(C v) { return this->ECylQ<C>::twoi(v); }
    __device__ C i1(C v) { return this->ECylQ<C>::i1(v); }
    __device__ C half(C v) { return this->ECylQ<C>::half(v); }
    __device__ C twohalf(C v) { return this->ECylQ<C>::twohalf(v); }
};
template <>
struct ECylF<double> {
    bool ok = true;
    double dx, dz, idx, idz, r2i, ri, r5, r25, i2i, ii, i5, i25;
    __device__ ECylF(const ECylArgs<double> &a, int i)
        : dx(a.dx), dz(a.dz), idx(a.idx), idz(a.idz) {
        r2i = 2. * double(i) * dx;
        ri = double(i) * dx;
        r5 = (double(i) + 0.5) * dx;
        r25 = 2. * (double(i) + 0.5) * dx;
        const long long s = a.nx2;
        i2i = a.inv[i];
        ii = a.inv[s + i];
        i5 = a.inv[2 * s + i];
        i25 = a.inv[3 * s + i];
    }
    __device__ double quot(double v, double d, double r) {
        const unsigned e = (unsigned)__double2hiint(v) & 0x7ff00000u;
        ok = ok && (e - ((1023u - 960u) << 20) < (1860u << 20) || v == 0.0);
        double q = __dmul_rn(v, r);
        q = __fma_rn(__fma_rn(-q, d, v), r, q);
        return __fma_rn(__fma_rn(-q, d, v), r, q);
    }
    __device__ double x(double v) { return quot(v, dx, idx); }
    __device__ double z(double v) { return quot(v, dz, idz); }
    __device__ double twoi(double v) { return quot(v, r2i, i2i); }
    __device__ double i1(double v) { return quot(v, ri, ii); }
    __device__ double half(double v) { return quot(v, r5, i5); }
    __device__ double twohalf(double v) { return quot(v, r25, i25); }
};

// 16 bytes of consecutive z cells, loaded and stored as one access (the
// pitch is a multiple of 32 cells and the first cell one of the vector's)
template <typename C>
struct ECylVec {
    static constexpr int V = 16 / (int)sizeof(C);
    C v[V];
    __device__ void ld(const C *p) {
        if constexpr (sizeof(C) == 4) {
            const float4 t = *reinterpret_cast<const float4 *>(p);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
            const double2 t = *reinterpret_cast<const double2 *>(p);
            v[0] = t.x; v[1] = t.y;
        }
    }
    // memory no launch writes
    __device__ void ldg(const C *p) {
        if constexpr (sizeof(C) == 4) {
            const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
            const double2 t = __ldg(reinterpret_cast<const double2 *>(p));
            v[0] = t.x; v[1] = t.y;
        }
    }
    __device__ void st(C *p) const {
        if constexpr (sizeof(C) == 4)
            *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
        else
            *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
    }
};

// column and row of single-cell thread t (ECylSplit), or false past the last
template <typename C>
__device__ __forceinline__ bool ecyl_single(const ECylArgs<C> &a, const ECylSplit &s, int t, int &i,
                                            int &j) {
    if (t < s.nfull) {   // column 0, then the columns from nx - 1 (or 1) on
        const int c = t / a.nz2;
        j = t - c * a.nz2;
        i = c == 0 ? 0 : (s.ja < s.jb ? a.nx - 2 + c : c);
        return true;
    }
    t -= s.nfull;
    if (s.ja == s.jb) return false;
    const int rows = a.nz2 - (s.jb - s.ja);   // rows outside [ja, jb) of columns 1 .. nx - 2
    const int c = t / rows;
    if (c >= a.nx - 2) return false;
    j = t - c * rows;
    if (j >= s.ja) j += s.jb - s.ja;
    i = 1 + c;
    return true;
}

struct ECylSrc {
    long long q;     // padded (pitched) cell
    int type;        // SM_SRC_FR / FT / FZ / BULK / KURKJIAN
    long long voff;  // first sample in vals
    int len;
};

struct ECylRec {
    int i, j;
    int comp;        // SM_VR ... or SM_DIV / SM_CURL
    int group;
    long long out;
};

// Sources and records that one of the two launches serves.  A source is added
// by the CTA that updates its cell, after the update: first[b] .. first[b + 1]
// are CTA b's, in the caller's order; mask: bit b mod 64 of the CTAs that have
// any.  The records are those of the fields the launch only reads, sampled by
// nblk CTAs of their own at the front of the grid: the stress launch takes the
// velocities (div and curl among them) of its step, the velocity launch the
// stresses of the step before.  Launches of their own were two of a step's four;
// with them gone and each launch overlapping the end of the one before, us per
// step: 2012 x 4024 FP32 mode 1 213 -> 174, 393 x 731 FP64 mode 0 41 -> 26.
struct ECylServe {
    unsigned long long mask;
    const int *first;
    const ECylSrc *src;
    const double *vals;
    long long it;            // the step whose samples the sources take
    int nblk, nrec;
    const ECylRec *rec;
    const int32_t *table;
    long long nsteps_max;
    double *traces;
    long long rec_it;        // the step the records sample
};

// a record's value; div and curl are formed in FP64 from the stored fields
// (their differences cancel, so FP32 arithmetic there would add error that
// the fields themselves do not carry)
template <typename C>
__device__ double ecyl_probe(const ECylArgs<C> &a, int comp, int i, int j) {
    auto F = [&](int k, int ii, int jj) -> double {
        return static_cast<double>(a.f[k][(long long)ii * a.pitch + jj]);
    };
    const double dx = static_cast<double>(a.dx), dz = static_cast<double>(a.dz);
    switch (comp) {
    case SM_VR: return F(C_VR, i, j);
    case SM_VT: return F(C_VT, i, j);
    case SM_VZ: return F(C_VZ, i, j);
    case SM_TRR: return F(C_TRR, i, j);
    case SM_TTT: return F(C_TTT, i, j);
    case SM_TZZ: return F(C_TZZ, i, j);
    case SM_TRZ: return F(C_TRZ, i, j);
    case SM_TRT: return F(C_TRT, i, j);
    case SM_TTZ: return F(C_TTZ, i, j);
    case SM_DIV: {
        // propagate.c:4090-4100, its radial term not divided by dr
        if (i + 1 >= a.nx2 || j + 1 >= a.nz2) return 0.0;
        return ((i + 1) * F(C_VR, i + 1, j) - i * F(C_VR, i, j)) / (i + 0.5) +
               a.n * F(C_VT, i, j) / ((i + 0.5) * dx) + (F(C_VZ, i, j + 1) - F(C_VZ, i, j)) / dz;
    }
    default: {   // curl, propagate.c:4102-4118
        if (j == 0) return 0.0;
        if (i == 0) {
            if (!(a.n % 2)) return 0.0;
            return (F(C_VR, i, j) - F(C_VR, i, j - 1)) / dz - (F(C_VZ, i, j) - -F(C_VZ, i, j)) / dx;
        }
        return (F(C_VR, i, j) - F(C_VR, i, j - 1)) / dz - (F(C_VZ, i, j) - F(C_VZ, i - 1, j)) / dx;
    }
    }
}

template <typename C>
__device__ __forceinline__ void ecyl_record(const ECylArgs<C> &a, const ECylServe &v, int r) {
    if (r >= v.nrec || v.rec_it >= v.nsteps_max) return;
    const ECylRec e = v.rec[r];
    const int32_t slot = v.table[(long long)e.group * v.nsteps_max + v.rec_it];
    if (slot >= 0) v.traces[e.out + slot] = ecyl_probe<C>(a, e.comp, e.i, e.j);
}

// CTA b's sources (two may share a cell: one thread, in order): forces add
// dt b * value (src.c:186-199), a Kurkjian source its value, scaled by dt on the
// host, to trr and tzz (src.c:231-236)
template <typename C>
__device__ __forceinline__ void ecyl_sources(const ECylArgs<C> &a, const ECylServe &v, int b) {
    if (!(v.mask >> (b & 63) & 1)) return;
    const int lo = v.first[b], hi = v.first[b + 1];
    if (lo == hi) return;
    __syncthreads();
    if (threadIdx.x) return;
    for (int k = lo; k < hi; ++k) {
        const ECylSrc s = v.src[k];
        if (v.it >= s.len) continue;
        const C x = static_cast<C>(v.vals[s.voff + v.it]);
        if (s.type == SM_SRC_FR || s.type == SM_SRC_BULK) a.f[C_VR][s.q] += a.m[CM_BJ][s.q] * x;
        if (s.type == SM_SRC_FT) a.f[C_VT][s.q] += a.m[CM_BIJ][s.q] * x;
        if (s.type == SM_SRC_FZ || s.type == SM_SRC_BULK) a.f[C_VZ][s.q] += a.m[CM_BI][s.q] * x;
        if (s.type == SM_SRC_KURKJIAN) {
            a.f[C_TRR][s.q] += x;
            a.f[C_TZZ][s.q] += x;
        }
    }
}

// the records of a run's last step, in a launch of their own
template <typename C>
__global__ void ecyl_gather_kernel(const __grid_constant__ ECylArgs<C> a, const __grid_constant__ ECylServe v) {
    ecyl_record<C>(a, v, blockIdx.x * blockDim.x + threadIdx.x);
}

// vr, vt, vz of cell (i, j): update_vr/vt/vz_cyl (mode 0) or *_cyl_n (n > 0)
template <typename C, bool NPOS>
__device__ void ecyl_velocity_cell(const ECylArgs<C> &a, int i, int j) {
    const ECylDev<C> d{a, i, j};
    const ECylQ<C> Q(a, i);
    const int n = a.n;
    const long long q = (long long)i * a.pitch + j;
    // vr: rows [0, nz2-1), columns from 1 (from 0 for odd n: the axis)
    if (j + 1 < a.nz2 && (i >= 1 || (NPOS && (n % 2)))) {
        C ddz = Q.z(d.G(C_TRZ, i, j + 1) - d.G(C_TRZ, i, j));
        if (d.zhalf()) ddz = d.zf_half(ZV_TRZ, ddz);
        C s;
        if (i == 0) {
            s = Q.x(d.G(C_TRR, i, j) - -d.G(C_TRR, i, j)) + ddz;
        } else if (i < a.nx) {
            const C A = Q.x(d.G(C_TRR, i, j) - d.G(C_TRR, i - 1, j));
            const C B = Q.twoi(d.G(C_TRR, i, j) + d.G(C_TRR, i - 1, j));
            const C D = Q.twoi(d.G(C_TTT, i, j) + d.G(C_TTT, i - 1, j));
            if (NPOS)
                s = A + B + Q.i1(C(n) * d.G(C_TRT, i, j)) - D + ddz;
            else
                s = A + B - D + ddz;
        } else {
            const C A = d.rf_node(RV_DTRR, Q.x(d.G(C_TRR, i, j) - d.G(C_TRR, i - 1, j)));
            const C B = d.rf_node(RV_TRR1, Q.twoi(d.G(C_TRR, i, j) + d.G(C_TRR, i - 1, j)));
            const C D = d.rf_node(RV_TTT1, Q.twoi(d.G(C_TTT, i, j) + d.G(C_TTT, i - 1, j)));
            if (NPOS) {
                const C E = d.rf_node(RV_TRT1, Q.i1(d.G(C_TRT, i, j)));
                s = A + B + C(n) * E - D + ddz;
            } else {
                s = A + B - D + ddz;
            }
        }
        a.f[C_VR][q] += d.M(CM_BJ) * s;
    }
    if (i + 1 < a.nx2) {
        // vt: rows [0, nz2-1)
        if (j + 1 < a.nz2) {
            C ddz = Q.z(d.G(C_TTZ, i, j + 1) - d.G(C_TTZ, i, j));
            if (d.zhalf()) ddz = d.zf_half(ZV_TTZ, ddz);
            const C A = Q.half(d.G(C_TRT, i + 1, j) + d.G(C_TRT, i, j));
            const C B = Q.x(d.G(C_TRT, i + 1, j) - d.G(C_TRT, i, j));
            C s;
            if (i + 1 < a.nx) {
                if (NPOS)
                    s = A + B - Q.half(C(n) * d.G(C_TTT, i, j)) + ddz;
                else
                    s = A + B + ddz;
            } else {
                const C fa = d.rf_half(RV_TRT2, A), fb = d.rf_half(RV_DTRT, B);
                if (NPOS) {
                    const C E = d.rf_half(RV_TTT2, Q.half(d.G(C_TTT, i, j)));
                    s = fa + fb - C(n) * E + ddz;
                } else {
                    s = fa + fb + ddz;
                }
            }
            a.f[C_VT][q] += d.M(CM_BIJ) * s;
        }
        // vz: rows from 1 (from 0 without a PML)
        if (j >= 1 || a.np == 0) {
            C ddz = Q.z(d.G(C_TZZ, i, j) - d.below(C_TZZ));
            if (d.znode()) ddz = d.zf_node(ZV_TZZ, ddz);
            const C A = Q.x(d.G(C_TRZ, i + 1, j) - d.G(C_TRZ, i, j));
            const C B = Q.twohalf(d.G(C_TRZ, i + 1, j) + d.G(C_TRZ, i, j));
            C s;
            if (i + 1 < a.nx) {
                if (NPOS)
                    s = ddz + A + B + Q.half(C(n) * d.G(C_TTZ, i, j));
                else
                    s = ddz + A + B;
            } else {
                const C fa = d.rf_half(RV_DTRZ, A), fb = d.rf_half(RV_TRZ, B);
                if (NPOS) {
                    const C E = d.rf_half(RV_TTZ, Q.half(d.G(C_TTZ, i, j)));
                    s = ddz + fa + fb + C(n) * E;
                } else {
                    s = ddz + fa + fb;
                }
            }
            a.f[C_VZ][q] += d.M(CM_BI) * s;
        }
    }
}

// The same for the vector of cells from (i, j) on, clear of every layer and
// edge; operation for operation the single cell's branch.  One cell per thread
// executed 286 instructions per cell (320 for the stresses), most of them
// addresses and layer tests, and was bound by issue and load latency; 16-byte
// accesses of four (FP32) or two (FP64) cells share both and leave the launch
// bound by HBM.  2020 x 4040 cells, FP32, mode 1: velocities 85 us against
// 151, stresses 109 against 176 (0.48 and 0.63 GB of DRAM traffic, 5.7 and
// 5.8 TB/s), 89 and 98 instructions per cell.  FP64, 1012 x 1024, mode 1: 61 us
// per step against 154.
template <typename C, bool NPOS>
__device__ __forceinline__ void ecyl_velocity_vec(const ECylArgs<C> &a, int i, int j) {
    using Vec = ECylVec<C>;
    constexpr int V = Vec::V;
    const long long q = (long long)i * a.pitch + j;
    const int p = a.pitch;
    Vec rr, rrm, tt, ttm, rz, rzp, rt, rtp, tz, zz, vr, vt, vz, bj, bi, bij;
    rr.ld(a.f[C_TRR] + q);
    rrm.ld(a.f[C_TRR] + q - p);
    tt.ld(a.f[C_TTT] + q);
    ttm.ld(a.f[C_TTT] + q - p);
    rz.ld(a.f[C_TRZ] + q);
    rzp.ld(a.f[C_TRZ] + q + p);
    rt.ld(a.f[C_TRT] + q);
    rtp.ld(a.f[C_TRT] + q + p);
    tz.ld(a.f[C_TTZ] + q);
    zz.ld(a.f[C_TZZ] + q);
    const C rz_n = a.f[C_TRZ][q + V], tz_n = a.f[C_TTZ][q + V];
    const C zz_b = a.f[C_TZZ][q - 1];
    vr.ld(a.f[C_VR] + q);
    vt.ld(a.f[C_VT] + q);
    vz.ld(a.f[C_VZ] + q);
    bj.ldg(a.m[CM_BJ] + q);
    bij.ldg(a.m[CM_BIJ] + q);
    bi.ldg(a.m[CM_BI] + q);
    const C n = C(a.n);
    Vec wr, wt, wz;
    auto update = [&](auto &Q) {
#pragma unroll
        for (int e = 0; e < V; ++e) {
            {
                const C ddz = Q.z((e + 1 < V ? rz.v[e + 1 < V ? e + 1 : e] : rz_n) - rz.v[e]);
                const C A = Q.x(rr.v[e] - rrm.v[e]);
                const C B = Q.twoi(rr.v[e] + rrm.v[e]);
                const C D = Q.twoi(tt.v[e] + ttm.v[e]);
                const C s = NPOS ? A + B + Q.i1(n * rt.v[e]) - D + ddz : A + B - D + ddz;
                wr.v[e] = vr.v[e] + bj.v[e] * s;
            }
            {
                const C ddz = Q.z((e + 1 < V ? tz.v[e + 1 < V ? e + 1 : e] : tz_n) - tz.v[e]);
                const C A = Q.half(rtp.v[e] + rt.v[e]);
                const C B = Q.x(rtp.v[e] - rt.v[e]);
                const C s = NPOS ? A + B - Q.half(n * tt.v[e]) + ddz : A + B + ddz;
                wt.v[e] = vt.v[e] + bij.v[e] * s;
            }
            {
                const C ddz = Q.z(zz.v[e] - (e > 0 ? zz.v[e > 0 ? e - 1 : 0] : zz_b));
                const C A = Q.x(rzp.v[e] - rz.v[e]);
                const C B = Q.twohalf(rzp.v[e] + rz.v[e]);
                const C s = NPOS ? ddz + A + B + Q.half(n * tz.v[e]) : ddz + A + B;
                wz.v[e] = vz.v[e] + bi.v[e] * s;
            }
        }
    };
    ECylF<C> F(a, i);
    update(F);
    if (sizeof(C) == 8 && !F.ok) {   // a numerator outside the quotients' range
        ECylQ<C> D(a, i);
        update(D);
    }
    wr.st(a.f[C_VR] + q);
    wt.st(a.f[C_VT] + q);
    wz.st(a.f[C_VZ] + q);
}

template <typename C, bool NPOS>
__global__ void __launch_bounds__(kECylThreads)
    ecyl_velocity_kernel(const __grid_constant__ ECylArgs<C> a, const ECylSplit s,
                         const __grid_constant__ ECylServe v) {
    chain_wait();
    chain_trigger();
    int b = blockIdx.x, i, j;
    if (b < v.nblk) {
        ecyl_record<C>(a, v, b * kECylThreads + (int)threadIdx.x);
        return;
    }
    b -= v.nblk;
    if (b < s.nsingle) {
        if (ecyl_single(a, s, b * kECylThreads + (int)threadIdx.x, i, j))
            ecyl_velocity_cell<C, NPOS>(a, i, j);
    } else {
        const int c = b - s.nsingle;
        i = 1 + c / s.nvb;
        const int l = (c % s.nvb) * kECylThreads + (int)threadIdx.x;
        if (l < s.nlane) ecyl_velocity_vec<C, NPOS>(a, i, s.ja + l * ECylVec<C>::V);
    }
    ecyl_sources<C>(a, v, b);
}

// trr ttt tzz, trz, trt, ttz of cell (i, j)
template <typename C, bool NPOS>
__device__ void ecyl_stress_cell(const ECylArgs<C> &a, int i, int j) {
    const ECylDev<C> d{a, i, j};
    const ECylQ<C> Q(a, i);
    const int n = a.n;
    const long long q = (long long)i * a.pitch + j;
    // trr, ttt, tzz: columns [0, nx2-1), rows [0, nz2-1)
    if (i + 1 < a.nx2 && j + 1 < a.nz2) {
        C dvrdr = Q.x(d.G(C_VR, i + 1, j) - d.G(C_VR, i, j));
        C vrr = Q.twohalf(d.G(C_VR, i + 1, j) + d.G(C_VR, i, j));
        C vtr = NPOS ? Q.half(d.G(C_VT, i, j)) : C(0);
        C dvzdz = Q.z(d.G(C_VZ, i, j + 1) - d.G(C_VZ, i, j));
        if (i + 1 >= a.nx) {
            dvrdr = d.rf_half(RV_DVR, dvrdr);
            vrr = d.rf_half(RV_VR1, vrr);
            if (NPOS) vtr = d.rf_half(RV_VT1, vtr);
        }
        if (d.zhalf()) dvzdz = d.zf_half(ZV_VZ, dvzdz);
        const C l2m = d.M(CM_L2M), l = d.M(CM_L);
        if (NPOS) {
            a.f[C_TRR][q] += l2m * dvrdr + l * (vrr + C(n) * vtr + dvzdz);
            a.f[C_TTT][q] += l2m * (vrr + C(n) * vtr) + l * (dvrdr + dvzdz);
            a.f[C_TZZ][q] += l2m * dvzdz + l * (dvrdr + vrr + C(n) * vtr);
        } else {
            a.f[C_TRR][q] += l2m * dvrdr + l * (vrr + dvzdz);
            a.f[C_TTT][q] += l2m * vrr + l * (dvrdr + dvzdz);
            a.f[C_TZZ][q] += l2m * dvzdz + l * (dvrdr + vrr);
        }
    }
    // trz (update_trz_cyl for every n): columns from 1, rows from 1
    if (i >= 1 && (j >= 1 || a.np == 0)) {
        C ddz = Q.z(d.G(C_VR, i, j) - d.below(C_VR));
        if (d.znode()) ddz = d.zf_trz(ddz);
        C ddr = Q.x(d.G(C_VZ, i, j) - d.G(C_VZ, i - 1, j));
        if (i >= a.nx) {
            const int ii = i - a.nx;
            ddr = d.cpml(d.rvar(RV_DVZ, ii), d.K(K_BHR_E, ii), d.K(K_CHR_E, ii),
                         d.K(K_IKHR_E, ii), ddr);
        }
        a.f[C_TRZ][q] += d.M(CM_MU) * (ddz + ddr);
    }
    // trt: columns from 1 (from 0 for odd n), every row
    if (i >= 1 || (NPOS && (n % 2))) {
        C s;
        if (i == 0) {
            s = Q.x(d.G(C_VT, i, j) - -d.G(C_VT, i, j));
        } else if (i < a.nx) {
            const C A = Q.x(d.G(C_VT, i, j) - d.G(C_VT, i - 1, j));
            const C D = Q.twoi(d.G(C_VT, i, j) + d.G(C_VT, i - 1, j));
            if (NPOS)
                s = A - Q.i1(C(n) * d.G(C_VR, i, j)) - D;
            else
                s = A - D;
        } else {
            const C A = d.rf_node(RV_DVT, Q.x(d.G(C_VT, i, j) - d.G(C_VT, i - 1, j)));
            const C D = d.rf_node(RV_VT2, Q.twoi(d.G(C_VT, i, j) + d.G(C_VT, i - 1, j)));
            if (NPOS) {
                const C B = d.rf_node(RV_VR2, Q.i1(d.G(C_VR, i, j)));
                s = A - C(n) * B - D;
            } else {
                s = A - D;
            }
        }
        a.f[C_TRT][q] += d.M(CM_MUJ) * s;
    }
    // ttz: columns [0, nx2-1), rows from 1 (from 0 without a PML)
    if (i + 1 < a.nx2 && (j >= 1 || a.np == 0)) {
        const C diff = d.G(C_VT, i, j) - d.below(C_VT);
        const C mui = d.M(CM_MUI);
        const bool zp = d.znode();
        if (!NPOS) {
            // interior rows: dt mui (vt_j - vt_j-1) / dz, the division last
            if (zp)
                a.f[C_TTZ][q] += mui * d.zf_node(ZV_VT, Q.z(diff));
            else
                a.f[C_TTZ][q] += Q.z(mui * diff);
        } else {
            const C ddz = zp ? d.zf_node(ZV_VT, Q.z(diff)) : Q.z(diff);
            C s;
            if (i + 1 < a.nx)
                s = ddz - Q.half(C(n) * d.G(C_VZ, i, j));
            else
                s = ddz - C(n) * d.rf_half(RV_VZ, Q.half(d.G(C_VZ, i, j)));
            a.f[C_TTZ][q] += mui * s;
        }
    }
}

// the same for the vector of cells from (i, j) on (see ecyl_velocity_vec)
template <typename C, bool NPOS>
__device__ __forceinline__ void ecyl_stress_vec(const ECylArgs<C> &a, int i, int j) {
    using Vec = ECylVec<C>;
    constexpr int V = Vec::V;
    const long long q = (long long)i * a.pitch + j;
    const int p = a.pitch;
    Vec vr, vrp, vt, vtm, vz, vzm, rr, tt, zz, rz, rt, tz, l2m, lam, mu, muj, mui;
    vr.ld(a.f[C_VR] + q);
    vrp.ld(a.f[C_VR] + q + p);
    vt.ld(a.f[C_VT] + q);
    vtm.ld(a.f[C_VT] + q - p);
    vz.ld(a.f[C_VZ] + q);
    vzm.ld(a.f[C_VZ] + q - p);
    const C vz_n = a.f[C_VZ][q + V];
    const C vr_b = a.f[C_VR][q - 1], vt_b = a.f[C_VT][q - 1];
    rr.ld(a.f[C_TRR] + q);
    tt.ld(a.f[C_TTT] + q);
    zz.ld(a.f[C_TZZ] + q);
    rz.ld(a.f[C_TRZ] + q);
    rt.ld(a.f[C_TRT] + q);
    tz.ld(a.f[C_TTZ] + q);
    l2m.ldg(a.m[CM_L2M] + q);
    lam.ldg(a.m[CM_L] + q);
    mu.ldg(a.m[CM_MU] + q);
    muj.ldg(a.m[CM_MUJ] + q);
    mui.ldg(a.m[CM_MUI] + q);
    const C n = C(a.n);
    Vec wrr, wtt, wzz, wrz, wrt, wtz;
    auto update = [&](auto &Q) {
#pragma unroll
        for (int e = 0; e < V; ++e) {
            {
                const C dvrdr = Q.x(vrp.v[e] - vr.v[e]);
                const C vrr = Q.twohalf(vrp.v[e] + vr.v[e]);
                const C dvzdz = Q.z((e + 1 < V ? vz.v[e + 1 < V ? e + 1 : e] : vz_n) - vz.v[e]);
                if (NPOS) {
                    const C vtr = Q.half(vt.v[e]);
                    wrr.v[e] = rr.v[e] + (l2m.v[e] * dvrdr + lam.v[e] * (vrr + n * vtr + dvzdz));
                    wtt.v[e] = tt.v[e] + (l2m.v[e] * (vrr + n * vtr) + lam.v[e] * (dvrdr + dvzdz));
                    wzz.v[e] = zz.v[e] + (l2m.v[e] * dvzdz + lam.v[e] * (dvrdr + vrr + n * vtr));
                } else {
                    wrr.v[e] = rr.v[e] + (l2m.v[e] * dvrdr + lam.v[e] * (vrr + dvzdz));
                    wtt.v[e] = tt.v[e] + (l2m.v[e] * vrr + lam.v[e] * (dvrdr + dvzdz));
                    wzz.v[e] = zz.v[e] + (l2m.v[e] * dvzdz + lam.v[e] * (dvrdr + vrr));
                }
            }
            {
                const C ddz = Q.z(vr.v[e] - (e > 0 ? vr.v[e > 0 ? e - 1 : 0] : vr_b));
                const C ddr = Q.x(vz.v[e] - vzm.v[e]);
                wrz.v[e] = rz.v[e] + (mu.v[e] * (ddz + ddr));
            }
            {
                const C A = Q.x(vt.v[e] - vtm.v[e]);
                const C D = Q.twoi(vt.v[e] + vtm.v[e]);
                const C s = NPOS ? A - Q.i1(n * vr.v[e]) - D : A - D;
                wrt.v[e] = rt.v[e] + (muj.v[e] * s);
            }
            {
                const C diff = vt.v[e] - (e > 0 ? vt.v[e > 0 ? e - 1 : 0] : vt_b);
                if (NPOS) {
                    const C ddz = Q.z(diff);
                    wtz.v[e] = tz.v[e] + (mui.v[e] * (ddz - Q.half(n * vz.v[e])));
                } else {
                    wtz.v[e] = tz.v[e] + (Q.z(mui.v[e] * diff));
                }
            }
        }
    };
    ECylF<C> F(a, i);
    update(F);
    if (sizeof(C) == 8 && !F.ok) {
        ECylQ<C> D(a, i);
        update(D);
    }
    wrr.st(a.f[C_TRR] + q);
    wtt.st(a.f[C_TTT] + q);
    wzz.st(a.f[C_TZZ] + q);
    wrz.st(a.f[C_TRZ] + q);
    wrt.st(a.f[C_TRT] + q);
    wtz.st(a.f[C_TTZ] + q);
}

template <typename C, bool NPOS>
__global__ void __launch_bounds__(kECylThreads)
    ecyl_stress_kernel(const __grid_constant__ ECylArgs<C> a, const ECylSplit s,
                         const __grid_constant__ ECylServe v) {
    chain_wait();
    chain_trigger();
    int b = blockIdx.x, i, j;
    if (b < v.nblk) {
        ecyl_record<C>(a, v, b * kECylThreads + (int)threadIdx.x);
        return;
    }
    b -= v.nblk;
    if (b < s.nsingle) {
        if (ecyl_single(a, s, b * kECylThreads + (int)threadIdx.x, i, j))
            ecyl_stress_cell<C, NPOS>(a, i, j);
    } else {
        const int c = b - s.nsingle;
        i = 1 + c / s.nvb;
        const int l = (c % s.nvb) * kECylThreads + (int)threadIdx.x;
        if (l < s.nlane) ecyl_stress_vec<C, NPOS>(a, i, s.ja + l * ECylVec<C>::V);
    }
    ecyl_sources<C>(a, v, b);
}

}  // namespace sm

using namespace sm;

struct sm_ecyl {
    int device = 0;
    int precision = SM_FP32;
    int nx = 0, nz = 0, np = 0, nx2 = 0, nz2 = 0, pitch = 0, n = 0;
    double dx = 0, dz = 0, dt = 0;
    size_t it = 0;
    size_t elem = 4;
    cudaStream_t stream = nullptr;
    DevBuf fields, mats, coef, zm, rm, inv;
    size_t fstride = 0;   // elements between fields
    // sources: forces (velocity launch) and the Kurkjian source (stress launch)
    struct Sources {
        unsigned long long mask = 0;
        DevBuf first, src, vals;
    } force, kurk;
    // records, and their copies by the launch that samples them
    std::vector<ECylRec> rec;
    SamplePlan plan;
    int nrec_v = 0, nrec_t = 0;   // velocities (div, curl), stresses
    DevBuf d_rec_v, d_rec_t, d_table, d_traces;
    KernelTimer timer;
};

namespace {

int ecyl_check(sm_ecyl_t h) {
    if (!h) return sm_fail(SM_EINVAL, "null e_cyl_iso handle");
    return SM_OK;
}

template <typename C>
ECylArgs<C> ecyl_args(sm_ecyl *h) {
    ECylArgs<C> a{};
    a.nx = h->nx;
    a.nz = h->nz;
    a.np = h->np;
    a.nx2 = h->nx2;
    a.nz2 = h->nz2;
    a.pitch = h->pitch;
    a.n = h->n;
    a.dx = static_cast<C>(h->dx);
    a.dz = static_cast<C>(h->dz);
    a.idx = static_cast<C>(1.0 / h->dx);
    a.idz = static_cast<C>(1.0 / h->dz);
    a.inv = h->inv.as<C>();
    C *f = h->fields.as<C>();
    for (int k = 0; k < 9; ++k) a.f[k] = f + (size_t)k * h->fstride;
    const C *m = h->mats.as<C>();
    for (int k = 0; k < 8; ++k) a.m[k] = m + (size_t)k * h->fstride;
    a.k = h->coef.as<C>();
    a.zm = h->zm.as<C>();
    a.rm = h->rm.as<C>();
    return a;
}

int ecyl_comp_ok(int c) {
    return c == SM_VR || c == SM_VT || c == SM_VZ || c == SM_TRR || c == SM_TTT || c == SM_TZZ ||
           c == SM_TRZ || c == SM_TRT || c == SM_TTZ || c == SM_DIV || c == SM_CURL;
}

int ecyl_field_of(int comp) {
    switch (comp) {
    case SM_VR: return C_VR;
    case SM_VT: return C_VT;
    case SM_VZ: return C_VZ;
    case SM_TRR: return C_TRR;
    case SM_TTT: return C_TTT;
    case SM_TZZ: return C_TZZ;
    case SM_TRZ: return C_TRZ;
    case SM_TRT: return C_TRT;
    case SM_TTZ: return C_TTZ;
    default: return -1;
    }
}

// the cells of the vector path (ECylSplit): columns 1 .. nx - 2 and the rows
// whose own and neighbouring values lie clear of both z layers and both edges
template <typename C>
ECylSplit ecyl_split(const sm_ecyl *h, int *nblocks) {
    constexpr int V = ECylVec<C>::V;
    ECylSplit s{};
    s.ja = (std::max(h->np, 1) + V - 1) / V * V;
    s.jb = (h->nz + h->np - 1) / V * V;   // rows below nz + np - 1
    long long full = h->nx2, rows = 0;    // no vector rows: every column whole
    // FP64 quotients (ECylF) want lengths far from the ends of the exponent range
    const bool sane = sizeof(C) == 4 || (std::min(h->dx, h->dz) > 1e-30 && std::max(h->dx, h->dz) < 1e30);
    if (sane && h->nx > 2 && s.jb > s.ja) {
        s.nlane = (s.jb - s.ja) / V;
        s.nvb = (s.nlane + kECylThreads - 1) / kECylThreads;
        full = 1 + (h->nx2 - (h->nx - 1));
        rows = (long long)(h->nz2 - (s.jb - s.ja)) * (h->nx - 2);
    } else {
        s.ja = s.jb = 0;
    }
    s.nfull = (int)(full * h->nz2);
    s.nsingle = (int)((full * h->nz2 + rows + kECylThreads - 1) / kECylThreads);
    *nblocks = s.nsingle + (s.nlane ? s.nvb * (h->nx - 2) : 0);
    return s;
}

// the CTA (past the record CTAs) that updates cell (i, j)
template <typename C>
int ecyl_block_of(const sm_ecyl *h, const ECylSplit &s, int i, int j) {
    if (s.nlane && i >= 1 && i <= h->nx - 2 && j >= s.ja && j < s.jb)
        return s.nsingle + (i - 1) * s.nvb + (j - s.ja) / ECylVec<C>::V / kECylThreads;
    long long t;
    if (!s.nlane) t = (long long)i * h->nz2 + j;
    else if (i == 0 || i >= h->nx - 1) t = (long long)(i == 0 ? 0 : i - (h->nx - 2)) * h->nz2 + j;
    else t = s.nfull + (long long)(i - 1) * (h->nz2 - (s.jb - s.ja)) + (j < s.ja ? j : j - (s.jb - s.ja));
    return (int)(t / kECylThreads);
}

// a launch's source tables; the list empty, or a failure: none
template <typename C>
int ecyl_set_list(sm_ecyl *h, sm_ecyl::Sources &S, const std::vector<ECylSrc> &src,
                  const std::vector<double> &vals) {
    S.mask = 0;
    if (src.empty()) return SM_OK;
    int nb = 0;
    const ECylSplit sp = ecyl_split<C>(h, &nb);
    unsigned long long mask = 0;
    std::vector<int> first(nb + 1, 0), at;
    auto block = [&](const ECylSrc &e) {
        return ecyl_block_of<C>(h, sp, (int)(e.q / h->pitch), (int)(e.q % h->pitch));
    };
    for (const ECylSrc &e : src) {
        const int b = block(e);
        first[b + 1]++;
        mask |= 1ull << (b & 63);
    }
    for (int b = 0; b < nb; ++b) first[b + 1] += first[b];
    at.assign(first.begin(), first.end() - 1);
    std::vector<ECylSrc> sorted(src.size());
    for (const ECylSrc &e : src) sorted[at[block(e)]++] = e;
    int rc;
    if ((rc = S.first.alloc(first.size() * sizeof(int))) || (rc = S.src.alloc(src.size() * sizeof(ECylSrc))) ||
        (rc = S.vals.alloc(std::max<size_t>(vals.size(), 1) * sizeof(double))))
        return rc;
    SM_CUDA_TRY(cudaMemcpyAsync(S.first.p, first.data(), S.first.bytes, cudaMemcpyHostToDevice, h->stream));
    SM_CUDA_TRY(cudaMemcpyAsync(S.src.p, sorted.data(), S.src.bytes, cudaMemcpyHostToDevice, h->stream));
    if (!vals.empty())
        SM_CUDA_TRY(cudaMemcpyAsync(S.vals.p, vals.data(), vals.size() * sizeof(double),
                                    cudaMemcpyHostToDevice, h->stream));
    SM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    S.mask = mask;   // (zero until the tables are complete)
    return SM_OK;
}

// what a launch serves: S's sources at step it, the records rec at step rec_it
ECylServe ecyl_serve(const sm_ecyl *h, const sm_ecyl::Sources &S, const DevBuf &rec, int nrec, long long it,
                     long long rec_it) {
    ECylServe v{};
    v.mask = S.mask;
    v.first = S.first.as<int>();
    v.src = S.src.as<ECylSrc>();
    v.vals = S.vals.as<double>();
    v.it = it;
    v.nrec = rec_it < 0 ? 0 : nrec;
    v.nblk = (v.nrec + kECylThreads - 1) / kECylThreads;
    v.rec = rec.as<ECylRec>();
    v.table = h->d_table.as<int32_t>();
    v.nsteps_max = (long long)h->plan.nsteps_max;
    v.traces = h->d_traces.as<double>();
    v.rec_it = rec_it;
    return v;
}

// steps of one run; the stress records of a step are sampled by the next
// step's velocity launch, the last step's after it
template <typename C>
int ecyl_steps(sm_ecyl *h, size_t nsteps) {
    const ECylArgs<C> a = ecyl_args<C>(h);
    int grd = 0;
    const ECylSplit sp = ecyl_split<C>(h, &grd);
    ChainTimer chain(h->timer, h->stream);
    for (size_t n = 0; n < nsteps; ++n) {
        const long long it = (long long)h->it;
        const ECylServe v = ecyl_serve(h, h->force, h->d_rec_t, h->nrec_t, it, n ? it - 1 : -1);
        const ECylServe t = ecyl_serve(h, h->kurk, h->d_rec_v, h->nrec_v, it, it);
        if (int rc = launch_chained(h->n > 0 ? ecyl_velocity_kernel<C, true> : ecyl_velocity_kernel<C, false>,
                                    grd + v.nblk, kECylThreads, 0, h->stream, a, sp, v))
            return rc;
        if (int rc = launch_chained(h->n > 0 ? ecyl_stress_kernel<C, true> : ecyl_stress_kernel<C, false>,
                                    grd + t.nblk, kECylThreads, 0, h->stream, a, sp, t))
            return rc;
        h->timer.launches += 2;
        h->it++;
        chain.n++;
    }
    chain.close();
    if (nsteps && h->nrec_t) {
        const ECylServe v = ecyl_serve(h, h->force, h->d_rec_t, h->nrec_t, 0, (long long)h->it - 1);
        ecyl_gather_kernel<C><<<v.nblk, kECylThreads, 0, h->stream>>>(a, v);
        h->timer.launches += 1;
    }
    return SM_OK;
}

template <typename C>
int upload_pitched(DevBuf &dst, size_t k, size_t stride, const double *src, int nx2, int nz2,
                   int pitch, cudaStream_t s) {
    std::vector<C> tmp((size_t)nx2 * pitch, C(0));
    for (int i = 0; i < nx2; ++i)
        for (int j = 0; j < nz2; ++j) tmp[(size_t)i * pitch + j] = static_cast<C>(src[(size_t)i * nz2 + j]);
    SM_CUDA_TRY(cudaMemcpyAsync(dst.as<C>() + k * stride, tmp.data(), tmp.size() * sizeof(C),
                                cudaMemcpyHostToDevice, s));
    SM_CUDA_TRY(cudaStreamSynchronize(s));
    return SM_OK;
}

}  // namespace

extern "C" size_t sm_ecyl_device_bytes(size_t nx, size_t nz, size_t np, int precision) {
    const size_t e = precision == SM_FP64 ? 8 : 4;
    const size_t nx2 = nx + np, nz2 = nz + 2 * np, pitch = round_up(nz2, 32);
    return e * (17 * nx2 * pitch + NZV * nx2 * (2 * np + 1) + NRV * (np + 1) * nz2 + 15 * (np + 1));
}

extern "C" int sm_ecyl_create(int device, size_t nx, size_t nz, size_t np, int n, double dx,
                              double dz, double dt, const double *const *mat,
                              const double *const *coef, int precision, sm_ecyl_t *out) {
    if (!out) return sm_fail(SM_EINVAL, "sm_ecyl_create: out is NULL");
    *out = nullptr;
    if (precision != SM_FP32 && precision != SM_FP64)
        return sm_fail(SM_EINVAL, "sm_ecyl_create: e_cyl_iso runs in FP32 or FP64 storage");
    if (nx < 2 || nz < 2 || n < 0 || !(dx > 0) || !(dz > 0) || !(dt > 0) || !mat || !coef)
        return sm_fail(SM_EINVAL, "sm_ecyl_create: bad argument");
    if (nx + np > 65535 || nz + 2 * np > (1u << 24))
        return sm_fail(SM_EINVAL, "sm_ecyl_create: grid too large (at most 65535 radial columns)");
    for (int k = 0; k < 8; ++k)
        if (!mat[k]) return sm_fail(SM_EINVAL, "sm_ecyl_create: material %d is NULL", k);
    for (int k = 0; k < 15; ++k)
        if (!coef[k]) return sm_fail(SM_EINVAL, "sm_ecyl_create: coefficient array %d is NULL", k);
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return sm_fail(SM_EINVAL, "sm_ecyl_create: no CUDA device %d", device);
    DeviceGuard g(device);
    std::unique_ptr<sm_ecyl> h(new (std::nothrow) sm_ecyl());
    if (!h) return sm_fail(SM_ENOMEM, "sm_ecyl_create: out of host memory");
    h->device = device;
    h->precision = precision;
    h->nx = (int)nx;
    h->nz = (int)nz;
    h->np = (int)np;
    h->nx2 = (int)(nx + np);
    h->nz2 = (int)(nz + 2 * np);
    h->pitch = (int)round_up((size_t)h->nz2, 32);
    h->n = n;
    h->dx = dx;
    h->dz = dz;
    h->dt = dt;
    h->elem = precision == SM_FP64 ? 8 : 4;
    SM_CUDA_TRY(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    h->fstride = (size_t)h->nx2 * h->pitch;
    int rc;
    if ((rc = h->fields.alloc(9 * h->fstride * h->elem))) return rc;
    if ((rc = h->mats.alloc(8 * h->fstride * h->elem))) return rc;
    if ((rc = h->coef.alloc((9 * np + 6 * (np + 1)) * h->elem + h->elem))) return rc;
    if ((rc = h->zm.alloc(NZV * (size_t)h->nx2 * (2 * np + 1) * h->elem))) return rc;
    if ((rc = h->rm.alloc(NRV * (np + 1) * (size_t)h->nz2 * h->elem))) return rc;
    if ((rc = h->fields.zero(h->stream)) || (rc = h->mats.zero(h->stream)) ||
        (rc = h->zm.zero(h->stream)) || (rc = h->rm.zero(h->stream)))
        return rc;
    // materials times dt, in FP64, then to the storage type
    std::vector<double> tmp((size_t)h->nx2 * h->nz2);
    for (int k = 0; k < 8; ++k) {
        for (size_t q = 0; q < tmp.size(); ++q) tmp[q] = dt * mat[k][q];
        rc = precision == SM_FP64
                 ? upload_pitched<double>(h->mats, k, h->fstride, tmp.data(), h->nx2, h->nz2, h->pitch, h->stream)
                 : upload_pitched<float>(h->mats, k, h->fstride, tmp.data(), h->nx2, h->nz2, h->pitch, h->stream);
        if (rc) return rc;
    }
    {   // per-column reciprocals of the radial lengths (ECylArgs::inv): formed in
        // FP64 from the expressions of ECylF, one rounding each
        const size_t nx2 = (size_t)h->nx2;
        std::vector<double> r(4 * nx2, 0.0);
        for (size_t i = 0; i < nx2; ++i) {
            r[i] = i ? 1.0 / (2. * i * dx) : 0.0;
            r[nx2 + i] = i ? 1.0 / (i * dx) : 0.0;
            r[2 * nx2 + i] = 1.0 / ((i + 0.5) * dx);
            r[3 * nx2 + i] = 1.0 / (2. * (i + 0.5) * dx);
        }
        if ((rc = h->inv.alloc(r.size() * h->elem))) return rc;
        rc = precision == SM_FP64 ? upload_convert<double>(h->inv.p, r.data(), r.size(), h->stream)
                                  : upload_convert<float>(h->inv.p, r.data(), r.size(), h->stream);
        if (rc) return rc;
    }
    std::vector<double> kt;
    for (int k = 0; k < 15; ++k) kt.insert(kt.end(), coef[k], coef[k] + (k < 9 ? np : np + 1));
    kt.push_back(0.0);
    rc = precision == SM_FP64 ? upload_convert<double>(h->coef.p, kt.data(), kt.size(), h->stream)
                              : upload_convert<float>(h->coef.p, kt.data(), kt.size(), h->stream);
    if (rc) return rc;
    SM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    *out = h.release();
    return SM_OK;
}

extern "C" int sm_ecyl_destroy(sm_ecyl_t h) {
    if (!h) return SM_OK;
    {
        DeviceGuard g(h->device);
        if (h->stream) cudaStreamSynchronize(h->stream);
        h->fields.release();
        h->mats.release();
        h->coef.release();
        h->zm.release();
        h->rm.release();
        h->inv.release();
        for (sm_ecyl::Sources *S : {&h->force, &h->kurk}) {
            S->first.release();
            S->src.release();
            S->vals.release();
        }
        h->d_rec_v.release();
        h->d_rec_t.release();
        h->d_table.release();
        h->d_traces.release();
        if (h->stream) cudaStreamDestroy(h->stream);
    }
    delete h;
    return SM_OK;
}

// Sources: force types (SM_SRC_FR, SM_SRC_FT, SM_SRC_FZ, SM_SRC_BULK) add
// dt b[index] fct[it] after the velocity update; one SM_SRC_KURKJIAN source
// adds dt fct[it] to trr and tzz after the stress update (the reference
// handles a Kurkjian first source alone, e_cyl_iso.c:497-502,664-666).
extern "C" int sm_ecyl_set_sources(sm_ecyl_t h, size_t nsrc, const size_t *index,
                                   const int *type, const double *fct, const size_t *length,
                                   size_t stride) {
    if (int rc = ecyl_check(h)) return rc;
    if (nsrc && (!index || !type || !fct || !length))
        return sm_fail(SM_EINVAL, "sm_ecyl_set_sources: NULL array");
    DeviceGuard g(h->device);
    const size_t N = (size_t)h->nx2 * h->nz2;
    std::vector<ECylSrc> force, kurk;
    std::vector<double> vals, kvals;
    for (size_t s = 0; s < nsrc; ++s) {
        if (index[s] >= N) return sm_fail(SM_EINVAL, "sm_ecyl_set_sources: source %zu outside the grid", s);
        if (length[s] > stride) return sm_fail(SM_EINVAL, "sm_ecyl_set_sources: length > stride");
        const long long q = (long long)(index[s] / h->nz2) * h->pitch + (long long)(index[s] % h->nz2);
        if (type[s] == SM_SRC_KURKJIAN) {
            if (!kurk.empty())
                return sm_fail(SM_EINVAL, "sm_ecyl_set_sources: one Kurkjian source at most");
            kurk.push_back(ECylSrc{q, type[s], 0, (int)length[s]});
            for (size_t t = 0; t < length[s]; ++t) kvals.push_back(h->dt * fct[s * stride + t]);
            continue;
        }
        if (type[s] != SM_SRC_FR && type[s] != SM_SRC_FT && type[s] != SM_SRC_FZ &&
            type[s] != SM_SRC_BULK)
            continue;   // the reference's cylindrical loop adds nothing for other types
        force.push_back(ECylSrc{q, type[s], (long long)vals.size(), (int)length[s]});
        vals.insert(vals.end(), fct + s * stride, fct + s * stride + length[s]);
    }
    SM_CUDA_TRY(cudaStreamSynchronize(h->stream));   // no step still reads the old tables
    const bool f64 = h->precision == SM_FP64;
    h->force.mask = h->kurk.mask = 0;   // a failure below leaves no sources
    int rc = f64 ? ecyl_set_list<double>(h, h->force, force, vals) : ecyl_set_list<float>(h, h->force, force, vals);
    if (!rc)
        rc = f64 ? ecyl_set_list<double>(h, h->kurk, kurk, kvals) : ecyl_set_list<float>(h, h->kurk, kurk, kvals);
    if (rc) h->force.mask = 0;
    return rc;
}

extern "C" int sm_ecyl_set_receivers(sm_ecyl_t h, size_t nrec, const size_t *index,
                                     const int *comp, const double *t0, const double *rdt,
                                     size_t nsteps_max) {
    if (int rc = ecyl_check(h)) return rc;
    if (nrec && (!index || !comp || !t0 || !rdt))
        return sm_fail(SM_EINVAL, "sm_ecyl_set_receivers: NULL array");
    DeviceGuard g(h->device);
    const size_t N = (size_t)h->nx2 * h->nz2;
    SamplePlan plan;   // a refused call leaves the handle's own records as they are
    if (int rc = plan.build(nrec, t0, rdt, h->dt, nsteps_max)) return rc;
    std::vector<ECylRec> rec, rv, rt;   // all, and by the launch that samples them
    long long out = 0;
    for (size_t r = 0; r < nrec; ++r) {
        if (index[r] >= N) return sm_fail(SM_EINVAL, "sm_ecyl_set_receivers: record %zu outside the grid", r);
        const int c = comp[r];
        if (!ecyl_comp_ok(c))
            return sm_fail(SM_EINVAL, "sm_ecyl_set_receivers: component %d of record %zu is not "
                                      "an e_cyl_iso component", c, r);
        const int grp = plan.group_of[r];
        rec.push_back(ECylRec{(int)(index[r] / h->nz2), (int)(index[r] % h->nz2), c, grp, out});
        const bool vel = c == SM_VR || c == SM_VT || c == SM_VZ || c == SM_DIV || c == SM_CURL;
        (vel ? rv : rt).push_back(rec.back());
        out += (long long)plan.count_total[grp];
    }
    h->rec.clear();   // a failure below leaves no records
    h->nrec_v = h->nrec_t = 0;
    int rc;
    if ((rc = h->d_traces.alloc(std::max<long long>(out, 1) * sizeof(double)))) return rc;
    if ((rc = h->d_traces.zero(h->stream))) return rc;
    if (nrec) {
        if ((rc = h->d_rec_v.alloc(rv.size() * sizeof(ECylRec)))) return rc;
        if ((rc = h->d_rec_t.alloc(rt.size() * sizeof(ECylRec)))) return rc;
        if ((rc = h->d_table.alloc(std::max<size_t>(plan.table.size(), 1) * sizeof(int32_t)))) return rc;
        if (!rv.empty())
            SM_CUDA_TRY(cudaMemcpyAsync(h->d_rec_v.p, rv.data(), h->d_rec_v.bytes, cudaMemcpyHostToDevice,
                                        h->stream));
        if (!rt.empty())
            SM_CUDA_TRY(cudaMemcpyAsync(h->d_rec_t.p, rt.data(), h->d_rec_t.bytes, cudaMemcpyHostToDevice,
                                        h->stream));
        if (!plan.table.empty())
            SM_CUDA_TRY(cudaMemcpyAsync(h->d_table.p, plan.table.data(), plan.table.size() * sizeof(int32_t),
                                        cudaMemcpyHostToDevice, h->stream));
    }
    SM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    h->nrec_v = (int)rv.size();
    h->nrec_t = (int)rt.size();
    h->rec.swap(rec);
    std::swap(h->plan, plan);
    return SM_OK;
}

extern "C" int sm_ecyl_run(sm_ecyl_t h, size_t nsteps) {
    if (int rc = ecyl_check(h)) return rc;
    DeviceGuard g(h->device);
    if (int rc = h->precision == SM_FP64 ? ecyl_steps<double>(h, nsteps) : ecyl_steps<float>(h, nsteps)) return rc;
    SM_CUDA_TRY(cudaGetLastError());
    return SM_OK;
}

extern "C" int sm_ecyl_sync(sm_ecyl_t h) {
    if (int rc = ecyl_check(h)) return rc;
    DeviceGuard g(h->device);
    SM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SM_OK;
}

extern "C" int sm_ecyl_reset(sm_ecyl_t h) {
    if (int rc = ecyl_check(h)) return rc;
    DeviceGuard g(h->device);
    int rc;
    if ((rc = h->fields.zero(h->stream)) || (rc = h->zm.zero(h->stream)) ||
        (rc = h->rm.zero(h->stream)) || (rc = h->d_traces.zero(h->stream)))
        return rc;
    SM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    h->it = 0;
    return SM_OK;
}

extern "C" int sm_ecyl_read_traces(sm_ecyl_t h, size_t rec0, size_t nrec, double *out,
                                   size_t ld, size_t *counts) {
    if (int rc = ecyl_check(h)) return rc;
    if (rec0 + nrec > h->rec.size())
        return sm_fail(SM_EINVAL, "sm_ecyl_read_traces: records [%zu, %zu) of %zu", rec0,
                       rec0 + nrec, h->rec.size());
    DeviceGuard g(h->device);
    SM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    const size_t lim = std::min(h->it, h->plan.nsteps_max);
    std::vector<size_t> gcount(h->plan.count_total.size(), 0);   // samples so far, per sampling group
    for (size_t g = 0; g < gcount.size(); ++g)
        for (size_t it = 0; it < lim; ++it)
            if (h->plan.table[g * h->plan.nsteps_max + it] >= 0) ++gcount[g];
    size_t need = 0, span = 0;   // samples so far, and the records' span on the device
    for (size_t r = 0; r < nrec; ++r) {
        const int g = h->rec[rec0 + r].group;
        if (counts) counts[r] = gcount[g];
        if (out && ld < gcount[g])
            return sm_fail(SM_EINVAL, "sm_ecyl_read_traces: ld %zu < %zu samples", ld, gcount[g]);
        need += gcount[g];
        span += h->plan.count_total[g];
    }
    if (!out || !need) return SM_OK;
    // The records are consecutive on the device: one copy, scattered into the
    // caller's rows (a copy per record costs about 7 us each: 24 records 0.43 ms),
    // unless most of it is samples not taken yet.
    if (span <= 4 * need) {
        std::unique_ptr<double[]> buf(new (std::nothrow) double[span]);
        if (!buf) return sm_fail(SM_ENOMEM, "sm_ecyl_read_traces: out of host memory");
        const long long at = h->rec[rec0].out;
        SM_CUDA_TRY(cudaMemcpy(buf.get(), h->d_traces.as<double>() + at, span * sizeof(double),
                               cudaMemcpyDeviceToHost));
        for (size_t r = 0; r < nrec; ++r)
            std::memcpy(out + r * ld, buf.get() + (h->rec[rec0 + r].out - at),
                        gcount[h->rec[rec0 + r].group] * sizeof(double));
        return SM_OK;
    }
    for (size_t r = 0; r < nrec; ++r)
        if (const size_t c = gcount[h->rec[rec0 + r].group])
            SM_CUDA_TRY(cudaMemcpy(out + r * ld, h->d_traces.as<double>() + h->rec[rec0 + r].out,
                                   c * sizeof(double), cudaMemcpyDeviceToHost));
    return SM_OK;
}

extern "C" int sm_ecyl_get_field(sm_ecyl_t h, int comp, double *out) {
    if (int rc = ecyl_check(h)) return rc;
    const int f = ecyl_field_of(comp);
    if (f < 0 || !out) return sm_fail(SM_EINVAL, "sm_ecyl_get_field: component %d", comp);
    DeviceGuard g(h->device);
    SM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    const size_t n = h->fstride;
    if (h->precision == SM_FP64) {
        std::vector<double> tmp(n);
        SM_CUDA_TRY(cudaMemcpy(tmp.data(), h->fields.as<double>() + f * n, n * sizeof(double),
                               cudaMemcpyDeviceToHost));
        for (int i = 0; i < h->nx2; ++i)
            for (int j = 0; j < h->nz2; ++j) out[(size_t)i * h->nz2 + j] = tmp[(size_t)i * h->pitch + j];
    } else {
        std::vector<float> tmp(n);
        SM_CUDA_TRY(cudaMemcpy(tmp.data(), h->fields.as<float>() + f * n, n * sizeof(float),
                               cudaMemcpyDeviceToHost));
        for (int i = 0; i < h->nx2; ++i)
            for (int j = 0; j < h->nz2; ++j) out[(size_t)i * h->nz2 + j] = tmp[(size_t)i * h->pitch + j];
    }
    return SM_OK;
}

extern "C" int sm_ecyl_set_field(sm_ecyl_t h, int comp, const double *in) {
    if (int rc = ecyl_check(h)) return rc;
    const int f = ecyl_field_of(comp);
    if (f < 0 || !in) return sm_fail(SM_EINVAL, "sm_ecyl_set_field: component %d", comp);
    DeviceGuard g(h->device);
    return h->precision == SM_FP64
               ? upload_pitched<double>(h->fields, f, h->fstride, in, h->nx2, h->nz2, h->pitch, h->stream)
               : upload_pitched<float>(h->fields, f, h->fstride, in, h->nx2, h->nz2, h->pitch, h->stream);
}

extern "C" int sm_ecyl_stream(sm_ecyl_t h, void **stream) {
    if (int rc = ecyl_check(h)) return rc;
    if (!stream) return sm_fail(SM_EINVAL, "sm_ecyl_stream: NULL");
    *stream = (void *)h->stream;
    return SM_OK;
}

extern "C" int sm_ecyl_set_timing(sm_ecyl_t h, int on) {
    if (int rc = ecyl_check(h)) return rc;
    DeviceGuard g(h->device);
    h->timer.set(on != 0);
    return SM_OK;
}

extern "C" int sm_ecyl_kernel_stats(sm_ecyl_t h, int reset, double *ms, size_t *timed,
                                    size_t *launches) {
    if (int rc = ecyl_check(h)) return rc;
    DeviceGuard g(h->device);
    return h->timer.stats(reset, ms, timed, launches);
}
