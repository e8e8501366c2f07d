// Fused structure-factor + adjoint kernel, second form (sm_103a): one body for
//   V = F2     FP32-bulk, two atoms per thread as packed FP32 pairs,
//   V = double the plain form, one atom per thread,
//   V = float  FP32-bulk, one atom per thread (multipole adjoint),
// over the symmetry forms (NSC operations in cosets of CS, sign group PAT).
//
// What bounds it, and why it is laid out so:
//   FP32: the FMA pipe and instruction issue.  A packed instruction (fma.f32x2) does two atoms in one issue slot
//     and holds the FMA pipe for two cycles, so the packed form halves the issue slots of everything that is the
//     same for both atoms: arithmetic, shared-memory reads of the reflection record (stored duplicated, {y, y}),
//     the reduction of F over the warp, loop and barrier work.  The code is kept in straight stretches: tiles with
//     and without l = 3, 4 harmonics run their own copy, and a group of four reflections without a line start runs
//     without a branch.  Against sf_grad_body (the same box): 5,000 isotropic atoms, P2_1 2_1 2_1, 54,704
//     reflections 1.70 -> 1.48 ms (189 warp instructions per two atoms and reflection instead of 2 x 167; the FMA
//     pipe 60% busy, two warps per scheduler); structure factors of 8,000 atoms, 100,003 reflections 3.97 -> 3.29 ms;
//     50,000 atoms, P4_3 2_1 2, multipole adjoint (V = float) 369 -> 300 ms; independent atoms, P2_1/c, 2,000 atoms,
//     50,021 reflections 0.46 -> 0.26 ms (one form factor for all operations: the transform of the phases alone, and
//     of an inversion pair only its real or imaginary half).
//   FP64: the FP64 pipe (about 1.6 lanes per clock and SM, 1/75 of FP32), so only the number of FP64 instructions
//     counts; integer work, shared-memory tables and loads are free beside it.  Exponentials and sines come from
//     shared-memory tables plus a short polynomial (exp_tab, sincos_tab), phases are exact 64-bit fixed point, and
//     every signed sum over a coset is a Walsh-Hadamard transform.  Against the earlier form (sf_grad_body in FP64,
//     66-90 FP64 instructions per atom, operation and reflection, now 28-65): P2_1, 2,501 isotropic atoms, 30,011
//     reflections 25.4 -> 10.5 ms; P4_3 2_1 2, 1,200 atoms, 20,011 reflections, multipole adjoint 34.7 -> 23.5 ms;
//     P2_1/c tabulated, 150 atoms, 20,021 reflections 1.58 -> 0.71 ms.  A block of four warps keeps its SM's FP64 pipe
//     busy, so registers and occupancy do not matter here.
// CEN: centrosymmetric structures whose inversion (at the origin) the engine takes have real adjoint weights and real
//   F: 6-9% less time than the general code (4,000 atoms, C2/c, FP32 1.07 -> 1.00 ms; 2,501 atoms, P2_1/c, FP64
//   11.05 -> 10.12 ms).
// Reflection records (pk_prep_kernel): per operation the integers of the exact phase (read at line starts only),
// per coset the harmonics, h' and its monomials of the coset's first operation.
#pragma once
#include "dsf_sf_kernel.cuh"

namespace dsf {

// ---------------------------------------------------------------------------
// the value of a thread: one atom (float, double) or two (F2)
// ---------------------------------------------------------------------------
struct F2 {
    float2 v;
};

template <typename V>
struct VTraits;
template <>
struct VTraits<F2> {
    using R = float;
    static constexpr int NA = 2;
};
template <>
struct VTraits<float> {
    using R = float;
    static constexpr int NA = 1;
};
template <>
struct VTraits<double> {
    using R = double;
    static constexpr int NA = 1;
};

__device__ __forceinline__ F2 vset(float a, float b) { return F2{make_float2(a, b)}; }
__device__ __forceinline__ F2 vneg(F2 a) { return F2{make_float2(-a.v.x, -a.v.y)}; }
__device__ __forceinline__ F2 vadd(F2 a, F2 b) { return F2{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 vsub(F2 a, F2 b) { return F2{__fadd2_rn(a.v, vneg(b).v)}; }
__device__ __forceinline__ F2 vmul(F2 a, F2 b) { return F2{__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) { return F2{__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ F2 vfnma(F2 a, F2 b, F2 c) { return F2{__ffma2_rn(vneg(a).v, b.v, c.v)}; }
__device__ __forceinline__ float vneg(float a) { return -a; }
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }
__device__ __forceinline__ float vmul(float a, float b) { return a * b; }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float vfnma(float a, float b, float c) { return fmaf(-a, b, c); }
__device__ __forceinline__ double vneg(double a) { return -a; }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double vfnma(double a, double b, double c) { return fma(-a, b, c); }
template <typename V>
__device__ __forceinline__ V vdup(typename VTraits<V>::R s)
{
    if constexpr (VTraits<V>::NA == 2) return vset(s, s);
    else return s;
}
// atom k of a value, and setting it
__device__ __forceinline__ float vget(F2 a, int k) { return k ? a.v.y : a.v.x; }
__device__ __forceinline__ float vget(float a, int) { return a; }
__device__ __forceinline__ double vget(double a, int) { return a; }
__device__ __forceinline__ void vput(F2 &a, int k, float s)
{
    if (k) a.v.y = s;
    else a.v.x = s;
}
__device__ __forceinline__ void vput(float &a, int, float s) { a = s; }
__device__ __forceinline__ void vput(double &a, int, double s) { a = s; }
// sum over the thread's atoms
__device__ __forceinline__ float vsum(F2 a) { return a.v.x + a.v.y; }
__device__ __forceinline__ float vsum(float a) { return a; }
__device__ __forceinline__ double vsum(double a) { return a; }

// ---------------------------------------------------------------------------
// FP64 functions from shared-memory tables
// ---------------------------------------------------------------------------
constexpr int kExpN = 1024;           // 2^(j / kExpN), j = 0 .. kExpN - 1
constexpr int kSinN = 512;            // sin(2 pi j / kSinN), j = 0 .. kSinN + kSinN / 4 - 1 (cosine: + kSinN / 4)
constexpr int kSinLen = kSinN + kSinN / 4;
constexpr int kMathTab = kExpN + kSinLen;  // doubles, [exp][sin]
// log2(e) kExpN as the sum of two doubles
constexpr double kExpHi = 1477.3197218702985, kExpLo = 2.0843800310713378e-14;

// e^x outside the table's range (|x| >= 512: near or past underflow or overflow, NaN)
static __device__ __noinline__ double exp_far(double x) { return exp(x); }

// e^x = 2^(n / kExpN) 2^(r / kExpN) in 8 FP64 instructions: n the nearest integer to x log2(e) kExpN (magic number),
// r the rest (one fused operation each for the constant's two parts, so r carries no rounding of the scaled
// argument), 2^(n / kExpN) from the table and the exponent, 2^(r / kExpN) by its Taylor polynomial of degree 3
// economised over |r| <= 1/2 (the quartic term's Chebyshev part folded into the quadratic: 7e-17 left).  The CUDA
// library's exp takes about twice as many.
__device__ __forceinline__ double exp_tab(double x, const double *tab)
{
    constexpr double c1 = 0.69314718055994530942 / kExpN;            // ln 2 / kExpN
    constexpr double a2 = (c1 * 0.5) * (c1 * 0.5);                    // (largest argument)^2
    constexpr double c2 = c1 * c1 * (0.5 + a2 / 24.0), c3 = c1 * c1 * c1 / 6.0;
    if ((__double2hiint(x) & 0x7fffffff) >= 0x40800000) return exp_far(x);
    const double magic = 6755399441055744.0;  // 1.5 2^52
    const double t = fma(x, kExpHi, magic);
    const int n = __double2loint(t);
    const double r = fma(x, kExpLo, fma(x, kExpHi, magic - t));
    const double tb = tab[n & (kExpN - 1)];
    const double p = r * fma(r, fma(r, c3, c2), c1);
    const double v = fma(tb, p, tb);  // in [1, 2); times 2^(n / kExpN) by integer addition to the exponent field
    return __hiloint2double(__double2hiint(v) + ((n >> 10) << 20), __double2loint(v));
}

// sin and cos of 2 pi P 2^-64: the nearest of kSinN directions from the table, the remainder (|x| <= pi / kSinN) by
// Taylor polynomials to x^5 and x^6 (truncation below 1e-17), and their product; 13 FP64 instructions
__device__ __forceinline__ void sincos_tab(uint64_t P, const double *tab, double *sn, double *cs)
{
    const uint32_t j = (uint32_t)((P + (1ull << 54)) >> 55) & (kSinN - 1);
    const int64_t r = (int64_t)(P - ((uint64_t)j << 55)) >> 3;  // |r| <= 2^51, units of 2^-61 turns
    const double x = (__longlong_as_double(0x4338000000000000ll + r) - 6755399441055744.0) *
                     (6.28318530717958647692 / 2305843009213693952.0);
    const double x2 = x * x;
    const double s = fma(x * x2, fma(x2, 1.0 / 120.0, -1.0 / 6.0), x);
    const double c = fma(x2, fma(x2, fma(x2, -1.0 / 720.0, 1.0 / 24.0), -0.5), 1.0);
    const double sj = tab[j], cj = tab[j + kSinN / 4];
    *sn = fma(sj, c, cj * s);
    *cs = fma(cj, c, -(sj * s));
}

// a float widened without the conversion unit (which runs at the FP64 rate): exponent re-biased and the mantissa
// moved by integer instructions; zero, subnormal, infinite and NaN values take the conversion
__device__ __forceinline__ double widen(float f)
{
    const uint32_t b = __float_as_uint(f);
    if (((b + 0x00800000u) & 0x7f000000u) == 0u) return (double)f;
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// FP32: sincos_fixed (sf_kernel.cuh) for every atom of the thread: P the phase in 2^32 fixed point per atom, lo the
// remainder in turns; the polynomials as packed operations
template <typename V>
__device__ __forceinline__ void sincos_fixed_v(const uint32_t (&P)[VTraits<V>::NA], V lo, V *sn, V *cs)
{
    constexpr int NA = VTraits<V>::NA;
    uint32_t q[NA];
    V r;
#pragma unroll
    for (int k = 0; k < NA; k++) {
        q[k] = (P[k] + 0x20000000u) >> 30;
        vput(r, k, (float)(int32_t)(P[k] - (q[k] << 30)));
    }
    const V th = vfma(r, vdup<V>(1.4629180792671596e-09f), vmul(vdup<V>(6.283185307179586f), lo));
    const V t2 = vmul(th, th);
    V sp = vfma(t2, vdup<V>(2.7557319e-06f), vdup<V>(-1.9841270e-04f));
    sp = vfma(t2, sp, vdup<V>(8.3333333e-03f));
    sp = vfma(t2, sp, vdup<V>(-1.6666667e-01f));
    const V sv = vfma(vmul(th, t2), sp, th);
    V cp = vfma(t2, vdup<V>(2.4801587e-05f), vdup<V>(-1.3888889e-03f));
    cp = vfma(t2, cp, vdup<V>(4.1666668e-02f));
    cp = vfma(t2, cp, vdup<V>(-0.5f));
    const V cv = vfma(t2, cp, vdup<V>(1.0f));
#pragma unroll
    for (int k = 0; k < NA; k++) {
        const float s1 = vget(sv, k), c1 = vget(cv, k);
        const float ss = (q[k] & 1u) ? c1 : s1, cc = (q[k] & 1u) ? s1 : c1;
        // the quadrant's signs on the sign bits
        vput(*sn, k, __uint_as_float(__float_as_uint(ss) ^ ((q[k] & 2u) << 30)));
        vput(*cs, k, __uint_as_float(__float_as_uint(cc) ^ (((q[k] + 1u) & 2u) << 30)));
    }
}

// ---------------------------------------------------------------------------
// reflection records
// ---------------------------------------------------------------------------
// per operation 32 bytes: FP32 {h' (3 ints), h.t in 2^32 fixed point; h' as floats}; FP64 {h' (3 ints); h.t in 2^64
// fixed point}
struct __align__(16) PkOp {
    int h[4];
    union {
        float hf[4];
        uint64_t tq;
    };
};
// per coset: slots of V's size (F2: duplicated): HC [25 harmonics][3 h'][6 monomials], other models [3 h'][6 monomials]
template <typename V>
__host__ __device__ constexpr int pk_slots(bool hc) { return sizeof(V) == 4 ? (hc ? 36 : 12) : (hc ? 34 : 10); }
template <typename V>
__host__ __device__ constexpr size_t pk_rec_bytes(bool hc, int ns, int ncosets)
{
    return sizeof(PkOp) * (size_t)ns + sizeof(V) * (size_t)pk_slots<V>(hc) * ncosets;
}

// a complex value, 16 bytes of record slots: one vector load each
template <typename V>
struct __align__(2 * sizeof(V)) PkPair {
    V re, im;
};
template <typename V>
struct __align__(16) PkV16 {
    V v[16 / sizeof(V)];
};

// parity classes gathered by character: index of parity class c in the coset's sign group (0 for CS = 1)
template <int CS, int PAT>
__host__ __device__ constexpr int pk_char(int c)
{
    return CS == 4 ? wht_char(PAT, c) : (CS == 2 ? parity3(c & PAT & 7) : 0);
}
__host__ __device__ constexpr int harmonic_l(int q) { return q < 1 ? 0 : q < 4 ? 1 : q < 9 ? 2 : q < 16 ? 3 : 4; }
// whether harmonic q is the first of its (l, character) slot; whether (l, character) has a harmonic
template <int CS, int PAT>
__host__ __device__ constexpr bool slot_first(int q)
{
    for (int p = harmonic_l(q) * harmonic_l(q); p < q; p++)
        if (pk_char<CS, PAT>(harmonic_class(p)) == pk_char<CS, PAT>(harmonic_class(q))) return false;
    return true;
}
template <int CS, int PAT>
__host__ __device__ constexpr bool slot_used(int l, int k)
{
    for (int p = l * l; p < (l + 1) * (l + 1); p++)
        if (pk_char<CS, PAT>(harmonic_class(p)) == k) return true;
    return false;
}

// Walsh-Hadamard transform over a coset (CS = 1, 2, 4)
template <int CS, typename V>
__device__ __forceinline__ void pk_wht(const V (&u)[CS], V (&W)[CS])
{
    if constexpr (CS == 1) {
        W[0] = u[0];
    } else if constexpr (CS == 2) {
        W[0] = vadd(u[0], u[1]);
        W[1] = vsub(u[0], u[1]);
    } else {
        const V t0 = vadd(u[0], u[1]), t1 = vsub(u[0], u[1]), t2 = vadd(u[2], u[3]), t3 = vsub(u[2], u[3]);
        W[0] = vadd(t0, t2);
        W[1] = vadd(t1, t3);
        W[2] = vsub(t0, t2);
        W[3] = vsub(t1, t3);
    }
}

// ---------------------------------------------------------------------------
// shared memory
// ---------------------------------------------------------------------------
template <typename V>
__host__ __device__ constexpr int pk_threads() { return kTileAtoms / VTraits<V>::NA; }
// line steps (and FP64 populations) in shared memory instead of registers
template <typename V, bool MP, bool ANISO, int NSC>
__host__ __device__ constexpr bool pk_step_smem()
{
    return NSC >= 8 || (VTraits<V>::NA == 2 ? ANISO && NSC >= 4 : sizeof(V) == 8 && MP);
}

template <typename V>
struct PkStage {
    size_t rs, tr, trm, gw, h2, cont, bytes, row;  // row: bytes of one type's rows (16 bytes of padding: no bank conflicts)
    __host__ __device__ PkStage(int ht, size_t rec, int max_types, bool mp, bool table)
    {
        using R = typename VTraits<V>::R;
        const int types = table ? 0 : max_types + 1;  // one more row, of zeros, for absent and excluded atoms
        row = sizeof(R) * 8 * (size_t)ht + 16;
        rs = 0;
        tr = rs + rec * (size_t)ht;
        trm = tr + row * types;
        gw = trm + (mp ? row * types : 0);
        h2 = gw + sizeof(R) * 2 * (size_t)ht;
        cont = h2 + sizeof(R) * (size_t)ht;
        bytes = (cont + sizeof(int) * (size_t)ht + 15) & ~(size_t)15;
    }
};

template <typename V, bool MP>
__host__ __device__ inline size_t pk_smem_bytes(int model, int ht, int nsc, int ncosets, int max_types, bool grad)
{
    using R = typename VTraits<V>::R;
    const bool hc = model == MODEL_HC;
    PkStage<V> L(ht, pk_rec_bytes<V>(hc, nsc, ncosets), max_types, MP, model == MODEL_TABLE);
    size_t b = 64 + 2 * L.bytes;
    b += sizeof(R) * 2 * (size_t)(pk_threads<V>() / 32) * ht;
    if (grad) b += sizeof(R) * 2 * (size_t)n_channels<R, MP>() * kTileAtoms;
    b += sizeof(int) * kMaxTileTypes;
    b += sizeof(R) == 8 ? sizeof(double) * kMathTab : 32 * (size_t)kTileAtoms;
    if (nsc >= 8 || (VTraits<V>::NA == 2 ? nsc >= 4 : sizeof(R) == 8 && MP)) b += 2 * sizeof(V) * (size_t)nsc * pk_threads<V>();
    if (sizeof(R) == 8 && hc) b += sizeof(V) * 25 * (size_t)pk_threads<V>();
    return b;
}

// The tiles of a structure for pk_kernel: kTileAtoms slots each, of atoms of one ADP kind, sorted so that a tile holds
// atoms with l >= 3 populations or none, and few types.  Two forms: dense, and (two atoms per thread, HC) pairs of
// slots 2t, 2t + 1 with atoms of one type each, a type with an odd count leaving one slot empty, so that a thread's
// two atoms share their radial terms.
struct PkTiles {
    const int *slot;    // [n_tiles][kTileAtoms] sorted atom index, -1: empty
    const int *ltype;   // [n_tiles][kTileAtoms] local type
    const int4 *info;   // [n_tiles] slots in use, types, highest l of the populations that are not zero, of all of them
    const int *types;   // [n_tiles][kMaxTileTypes]
    int n_plain;        // tiles below it hold atoms without anisotropic ADPs
    int max_types;
};

template <typename R>
struct PkEight {
    R v[8];
};
template <int N>
struct PkInt {
    static constexpr int value = N;
};
struct PkYes {
    static constexpr bool value = true;
};
struct PkNo {
    static constexpr bool value = false;
};

struct PkLaunch {
    int hkl_chunk, ht, n_hkl_pad;
    int n_chunks;          // reflection chunks of a tile (pk_kernel)
    PkTiles T;
    const void *pk;        // reflection records
    const void *tr, *trm;  // R [n_types][n_hkl_pad][8]
    const int *cont;
    const double *math;    // kMathTab doubles (FP64)
    int *error, stall_first;
};

template <typename V, int MODEL, bool MP, bool ANISO, int NSC, int CS, bool GRAD, bool INV, int PAT, bool CEN, bool ROLL,
          bool HL>
__device__ __forceinline__ void pk_body(const DevStructure &S, const CallBuffers &C, const PkLaunch &L, const int tile,
                                        const int chunk)
{
    using R = typename VTraits<V>::R;
    using R2 = typename Vec2<R>::T;
    using V2 = PkPair<V>;
    constexpr int NA = VTraits<V>::NA;
    constexpr bool F64 = sizeof(R) == 8;
    constexpr bool HC = MODEL == MODEL_HC, TABLE = MODEL == MODEL_TABLE, IAM = MODEL == MODEL_IAM;
    constexpr int NC = NSC / CS, NZ = INV ? NSC / 2 : NSC;
    constexpr bool INVC = INV && CS == NSC && CS > 1;  // the images lie in the same coset
    constexpr int NT = n_channels<R, MP>();
    constexpr int NL = HL ? 5 : 3, NH = NL * NL;  // levels of the angular sums (HL: l = 3, 4 too), harmonics
    constexpr bool SAME = HC && NA == 2;          // a thread's atoms share their type
    constexpr int TH = pk_threads<V>(), WARPS = TH / 32;
    constexpr bool STEP_SM = pk_step_smem<V, MP, ANISO, NSC>(), PG_SM = F64 && HC;
    constexpr int SLOTS = pk_slots<V>(HC);
    constexpr size_t REC = pk_rec_bytes<V>(HC, NSC, NC);
    constexpr int HOFF = HC ? 25 : 0;
    constexpr bool ROLL_J = NSC > 4 || MP || F64 || ROLL;
    // FP32 with many cosets: a reflection's position and ADP derivatives are summed over the cosets apart, one rounding
    // into the running sum instead of one per coset (P4_3 2_1 2, independent atoms, 2,000 atoms, 50,021 reflections: d_xyz
    // 1.8e-7 from 64 bits, without 3.1e-7; 1,089 -> 1,130 us)
    constexpr bool OWN = !F64 && GRAD && NC >= 4;
    static_assert(NSC % CS == 0 && (CS == 1 || CS == 2 || CS == 4), "cosets of one, two or four");
    static_assert(!INV || (!HC && NSC % 2 == 0), "inversion pairs: generic models");
    static_assert(GRAD || !MP, "the multipole adjoint needs the derivative pass");
    static_assert(!TABLE || F64, "FP32 tabulated structures take sf_grad_body");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int ht = L.ht;
    const int h_begin = chunk * L.hkl_chunk;
    const int h_end = min(S.n_hkl, h_begin + L.hkl_chunk);
    if (h_begin >= h_end) return;
    const int4 info = L.T.info[tile];
    const int n_at = info.x, nT = info.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw);
    const PkStage<V> SL(ht, REC, L.T.max_types, MP, TABLE);
    unsigned char *stage0 = smem_raw + 64;
    R2 *sF = reinterpret_cast<R2 *>(stage0 + 2 * SL.bytes);  // [warps of a part][ht]
    R *sTot = reinterpret_cast<R *>(sF + WARPS * ht);        // [NT][kTileAtoms], Kahan total and compensation
    R *sCmp = sTot + (GRAD ? NT * kTileAtoms : 0);
    unsigned char *sp = reinterpret_cast<unsigned char *>(sCmp + (GRAD ? NT * kTileAtoms : 0));
    double *sMath = reinterpret_cast<double *>(sp);
    if constexpr (F64) sp += sizeof(double) * kMathTab;
    V2 *sStep = reinterpret_cast<V2 *>(sp);  // [NSC][TH]
    if constexpr (STEP_SM) sp += 2 * sizeof(V) * NSC * TH;
    V *sPg = reinterpret_cast<V *>(sp);    // [25][TH]
    if constexpr (PG_SM) sp += sizeof(V) * 25 * TH;
    int4 *sX = reinterpret_cast<int4 *>(sp);  // FP32: fixed-point positions and their remainders (read at anchors)
    float4 *sXl = reinterpret_cast<float4 *>(sX + kTileAtoms);
    if constexpr (!F64) sp += 32 * kTileAtoms;
    int *sTypes = reinterpret_cast<int *>(sp);

    // Small tiles: the block's threads in `split` parts of TH / split atom slots, each part taking its own stretch of
    // every sub-tile, so a tile of few atoms still uses every warp and every FP64 sub-unit.  FP64: parts of eight lanes
    // and more, of any stretch (an FP64 instruction costs the same however many lanes are in use: 32 atoms, P2_1/c,
    // host call 172 -> 157 us).  FP32: whole warps and stretches of four reflections (the straight code's group);
    // smaller ones start every stretch at an exact phase and add eight parts' derivatives by atomics (20 atoms, P-1,
    // one call after another on a stream: 32 us, with parts of eight lanes 40; the constant width also takes 5,000
    // isotropic atoms of P2_1 2_1 2_1 from 1.54 to 1.49 ms)
    constexpr int MIN_SLOTS = F64 ? 8 : 32, MIN_SEG = F64 ? 1 : 4;
    int slots = TH;
    while (slots > MIN_SLOTS && slots / 2 * NA >= n_at && ht * slots / 2 >= MIN_SEG * TH) slots >>= 1;
    const int split = TH / slots, part_id = tid / slots, slot = tid - part_id * slots;
    const int width = F64 ? min(slots, 32) : 32, wrow = slot / 32;  // lanes of a part inside a warp, the warp's row of sF
    const int seg = ht / split, seg0 = part_id * seg;  // this thread's reflections of a sub-tile: [seg0, seg0 + seg)

    for (int i = tid; i < nT; i += TH) sTypes[i] = L.T.types[tile * kMaxTileTypes + i];
    if constexpr (GRAD) {
        for (int q = tid; q < NT * kTileAtoms; q += TH) {
            sTot[q] = R(0);
            sCmp[q] = R(0);
        }
    }
    if constexpr (F64) {
        for (int q = tid; q < kMathTab; q += TH) sMath[q] = L.math[q];
    }
    if constexpr (!TABLE) {
        for (int q = tid; q < 2 * (int)(SL.row / 16); q += TH) {  // the zero rows of both stages
            unsigned char *st = stage0 + (q & 1) * SL.bytes + SL.row * L.T.max_types;
            reinterpret_cast<int4 *>(st + SL.tr)[q >> 1] = make_int4(0, 0, 0, 0);
            if constexpr (MP) reinterpret_cast<int4 *>(st + SL.trm)[q >> 1] = make_int4(0, 0, 0, 0);
        }
    }
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncthreads();

    const unsigned char *pk_g = reinterpret_cast<const unsigned char *>(L.pk);
    const R *tr_g = reinterpret_cast<const R *>(L.tr), *trm_g = reinterpret_cast<const R *>(L.trm);
    const R2 *gw_g;
    const R *h2_g;
    if constexpr (F64) {
        gw_g = C.gw_d;
        h2_g = S.h2;
    } else {
        gw_g = C.gw_f;
        h2_g = S.h2f;
    }

    // warp 0 streams a sub-tile into one stage buffer (TMA bulk copies; a lane per type's rows)
    auto issue = [&](int buf, int h0) {
        unsigned char *st = stage0 + buf * SL.bytes;
        const uint32_t rs_bytes = (uint32_t)(REC * ht), tr_bytes = (uint32_t)(sizeof(R) * 8 * ht);
        fence_proxy_async();
        if (lane == 0)
            mbar_expect_tx(&bar[buf], rs_bytes + (uint32_t)((3 * sizeof(R) + sizeof(int)) * ht) +
                                          (TABLE ? 0u : tr_bytes * nT * (MP ? 2u : 1u)));
        __syncwarp();
        if constexpr (!TABLE) {
            for (int t = lane; t < nT; t += 32) {
                const size_t row = ((size_t)sTypes[t] * L.n_hkl_pad + h0) * 8;
                bulk_copy(st + SL.tr + SL.row * t, tr_g + row, tr_bytes, &bar[buf]);
                if constexpr (MP) bulk_copy(st + SL.trm + SL.row * t, trm_g + row, tr_bytes, &bar[buf]);
            }
        }
        if (lane == 0) {
            bulk_copy(st + SL.rs, pk_g + REC * (size_t)h0, rs_bytes, &bar[buf]);
            bulk_copy(st + SL.gw, gw_g + h0, (uint32_t)(2 * sizeof(R) * ht), &bar[buf]);
            bulk_copy(st + SL.h2, h2_g + h0, (uint32_t)(sizeof(R) * ht), &bar[buf]);
            bulk_copy(st + SL.cont, L.cont + h0, (uint32_t)(sizeof(int) * ht), &bar[buf]);
        }
    };
    if (warp == 0 && !L.stall_first) issue(0, h_begin);

    // the thread's atoms; absent and excluded ones are all zeros (their radial rows too), so they add nothing
    V w = vdup<V>(R(0)), anre = w, anim = w, pg[HC && !PG_SM ? NH : 1], adp[ANISO ? 6 : 1];
    V step_re[STEP_SM ? 1 : NZ], step_im[STEP_SM ? 1 : NZ], e_re[NZ], e_im[NZ];
    uint64_t xq64[3] = {0, 0, 0};
    int atom[NA];
    uint32_t toff[SAME ? 1 : NA];  // offset of the atom's radial rows inside a stage's table
    bool active[NA];
#pragma unroll
    for (int q = 0; q < (HC && !PG_SM ? NH : 1); q++) pg[q] = vdup<V>(R(0));
#pragma unroll
    for (int q = 0; q < (ANISO ? 6 : 1); q++) adp[q] = vdup<V>(R(0));
#pragma unroll
    for (int s = 0; s < NZ; s++) { e_re[s] = vdup<V>(R(1)); e_im[s] = vdup<V>(R(0)); }
#pragma unroll
    for (int s = 0; s < (STEP_SM ? 1 : NZ); s++) { step_re[s] = vdup<V>(R(1)); step_im[s] = vdup<V>(R(0)); }
    bool any = false;
#pragma unroll
    for (int k = 0; k < NA; k++) {
        const int la = slot * NA + k;
        atom[k] = la < n_at ? L.T.slot[tile * kTileAtoms + la] : -1;
        const size_t a = (size_t)max(atom[k], 0);
        active[k] = atom[k] >= 0 && S.atom_active[a] != 0;
        if (!SAME || k == 0) toff[SAME ? 0 : k] = (uint32_t)SL.row * L.T.max_types;
        if constexpr (!F64) {
            sX[k * TH + tid] = make_int4(0, 0, 0, 0);
            sXl[k * TH + tid] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if constexpr (PG_SM)
            for (int q = 0; q < NH; q++) sPg[q * TH + tid] = active[k] ? S.atom_pg_d[25 * a + q] : 0.0;
        if constexpr (STEP_SM)
            for (int s = 0; s < NSC; s++) {
                R2 st;
                st.x = R(1);
                st.y = R(0);
                if (active[k]) {
                    if constexpr (F64) st = S.atom_step_d[a * NSC + s];
                    else st = S.atom_step_f[a * NSC + s];
                }
                vput(sStep[s * TH + tid].re, k, st.x);
                vput(sStep[s * TH + tid].im, k, st.y);
            }
        if (!active[k]) continue;
        any = true;
        // (an excluded partner of a pair keeps zero populations, weight and dispersion, so the shared rows add nothing)
        if constexpr (!TABLE) toff[SAME ? 0 : k] = (uint32_t)SL.row * L.T.ltype[tile * kTileAtoms + la];
        if constexpr (F64) {
            w = S.atom_w_d[a];
            const double2 an = S.atom_anom_d[a];
            anre = an.x;
            anim = an.y;
#pragma unroll
            for (int q = 0; q < (ANISO ? 6 : 1); q++) adp[q] = -S.atom_adp_d[6 * a + q];
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const double x = S.atom_xd[3 * a + j];
                xq64[j] = __double2ull_rn((x - floor(x)) * 18446744073709551616.0);
            }
        } else {
            vput(w, k, S.atom_w_f[a]);
            const float2 an = S.atom_anom_f[a];
            vput(anre, k, an.x);
            vput(anim, k, an.y);
#pragma unroll
            for (int q = 0; q < (ANISO ? 6 : 1); q++) vput(adp[q], k, -S.atom_adp_f[6 * a + q]);
            sX[k * TH + tid] = make_int4((int)S.atom_xq[3 * a], (int)S.atom_xq[3 * a + 1], (int)S.atom_xq[3 * a + 2], 0);
            sXl[k * TH + tid] = make_float4(S.atom_xlo[3 * a], S.atom_xlo[3 * a + 1], S.atom_xlo[3 * a + 2], 0.f);
            if constexpr (HC) {
#pragma unroll
                for (int q = 0; q < NH; q++) vput(pg[q], k, S.atom_pg_f[25 * a + q]);
            }
        }
        if constexpr (!STEP_SM) {
#pragma unroll
            for (int s = 0; s < NZ; s++) {
                R2 st;
                if constexpr (F64) st = S.atom_step_d[a * NSC + s];
                else st = S.atom_step_f[a * NSC + s];
                vput(step_re[s], k, st.x);
                vput(step_im[s], k, st.y);
            }
        }
    }
    const bool warp_any = __any_sync(0xffffffffu, any);  // a warp without atoms only takes part in the barriers

    uint32_t parity[2] = {0u, 0u};
    V part[NT];
#pragma unroll
    for (int q = 0; q < NT; q++) part[q] = vdup<V>(R(0));
    const int fold = max(1, 32 * split / ht);  // partial sums of about 32 reflections per compensated addition
    int k_sub = 0;
    for (int h0 = h_begin; h0 < h_end; h0 += ht, k_sub++) {
        const int buf = k_sub & 1;
        if (warp == 0 && h0 + ht < h_end) issue(buf ^ 1, h0 + ht);
        const uint32_t phase = parity[buf];
        const bool ok = mbar_wait(&bar[buf], phase);
        parity[buf] ^= 1u;
        // (the barrier also keeps the block's warps at the same code: without it they run 2% slower)
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicOr(L.error, 1);
                // bounded: let this sub-tile's copies and the next one's (if issued) land first
                mbar_wait(&bar[buf], phase);
                if (h0 + ht < h_end) mbar_wait(&bar[buf ^ 1], parity[buf ^ 1]);
            }
            return;
        }
        const unsigned char *st = stage0 + buf * SL.bytes;
        const R2 *sG = reinterpret_cast<const R2 *>(st + SL.gw);
        const R *sH2 = reinterpret_cast<const R *>(st + SL.h2);
        const int *sCont = reinterpret_cast<const int *>(st + SL.cont);

        // the first reflection of a stretch: with several parts each stretch is apart from the one before
        const bool fresh = split > 1 || k_sub == 0;
        // reflection hl of the sub-tile: its partial F over the thread's atoms in (fr, fi)
        auto reflection = [&](const int hl, auto may_anchor, R &fr_out, R &fi_out) {
            const unsigned char *rec = st + SL.rs + REC * (size_t)hl;
            const PkOp *ops = reinterpret_cast<const PkOp *>(rec);
            const V *cos_rec = reinterpret_cast<const V *>(rec + sizeof(PkOp) * NSC);
            // ---- phases: exact at line and stretch starts, one complex multiplication per operation in between
            if (decltype(may_anchor)::value && ((sCont[hl] & (F64 ? 2 : 1)) == 0 || (hl == seg0 && fresh))) {
#pragma unroll
                for (int s = 0; s < NZ; s++) {
                    const PkOp op = ops[s];
                    if constexpr (F64) {
                        const uint64_t P = (uint64_t)(int64_t)op.h[0] * xq64[0] + (uint64_t)(int64_t)op.h[1] * xq64[1] +
                                           (uint64_t)(int64_t)op.h[2] * xq64[2] + op.tq;
                        sincos_tab(P, sMath + kExpN, &e_im[s], &e_re[s]);
                    } else {
                        uint32_t P[NA];
                        V lo;
#pragma unroll
                        for (int k = 0; k < NA; k++) {
                            const int4 xv = sX[k * TH + tid];
                            P[k] = (uint32_t)op.h[0] * (uint32_t)xv.x + (uint32_t)op.h[1] * (uint32_t)xv.y +
                                   (uint32_t)op.h[2] * (uint32_t)xv.z + (uint32_t)op.h[3];
                        }
#pragma unroll
                        for (int k = 0; k < NA; k++) {
                            const float4 xl = sXl[k * TH + tid];
                            vput(lo, k, op.hf[0] * xl.x + op.hf[1] * xl.y + op.hf[2] * xl.z);
                        }
                        sincos_fixed_v<V>(P, lo, &e_im[s], &e_re[s]);
                    }
                }
            } else {
#pragma unroll
                for (int s = 0; s < NZ; s++) {
                    V sr, si;
                    if constexpr (STEP_SM) {
                        const V2 sv = sStep[s * TH + tid];
                        sr = sv.re;
                        si = sv.im;
                    } else {
                        sr = step_re[s];
                        si = step_im[s];
                    }
                    const V cs = vfnma(e_im[s], si, vmul(e_re[s], sr));
                    e_im[s] = vfma(e_im[s], sr, vmul(e_re[s], si));
                    e_re[s] = cs;
                }
            }
            // ---- radial terms, isotropic temperature factor, adjoint weight
            const R2 g = sG[hl];
            V fs = anre, r[5];
            if constexpr (!TABLE) {
                constexpr int NR = SAME ? 1 : NA;
                R rr[NR][6];
#pragma unroll
                for (int k = 0; k < NR; k++) {
                    const R *rad = reinterpret_cast<const R *>(st + SL.tr + toff[k]) + 8 * hl;
                    if constexpr (IAM) {
                        rr[k][0] = rad[0];
                    } else if constexpr (F64) {
                        const double2 ra = reinterpret_cast<const double2 *>(rad)[0];
                        const double2 rb = reinterpret_cast<const double2 *>(rad)[1];
                        const double2 rc = reinterpret_cast<const double2 *>(rad)[2];
                        rr[k][0] = ra.x; rr[k][1] = ra.y; rr[k][2] = rb.x; rr[k][3] = rb.y; rr[k][4] = rc.x; rr[k][5] = rc.y;
                    } else {
                        const float4 ra = reinterpret_cast<const float4 *>(rad)[0];
                        const float2 rb = reinterpret_cast<const float2 *>(rad)[2];
                        rr[k][0] = ra.x; rr[k][1] = ra.y; rr[k][2] = ra.z; rr[k][3] = ra.w; rr[k][4] = rb.x; rr[k][5] = rb.y;
                    }
                }
                V f0;
#pragma unroll
                for (int k = 0; k < NA; k++) vput(f0, k, rr[k % NR][0]);
                fs = vadd(fs, f0);
                if constexpr (HC) {
#pragma unroll
                    for (int l = 0; l < NL; l++)
#pragma unroll
                        for (int k = 0; k < NA; k++) vput(r[l], k, rr[k % NR][1 + l]);
                }
            }
            // CEN: an inversion at the origin, taken by the engine: F is twice the real part, the adjoint weight real
            V Tiso = vdup<V>(R(1)), gre = vdup<V>(g.x), gim = vdup<V>(CEN ? R(0) : g.y);
            auto texp_v = [&](V x) -> V {
                if constexpr (F64) {
                    return exp_tab(x, sMath);
                } else {
                    V t;
#pragma unroll
                    for (int k = 0; k < NA; k++) vput(t, k, texp<float>(vget(x, k)));
                    return t;
                }
            };
            if constexpr (!ANISO) {
                Tiso = texp_v(vmul(adp[0], vdup<V>(sH2[hl])));
                if constexpr (GRAD && !IAM) {
                    gre = vmul(gre, Tiso);
                    if constexpr (!CEN) gim = vmul(gim, Tiso);
                }
            }
            V gfr = gre, gfi = gim;  // IAM: g f T (one form factor for every operation)
            V fTr = fs, fTi = anim;
            if constexpr (IAM) {
                if constexpr (!ANISO) {
                    fTr = vmul(fs, Tiso);
                    fTi = vmul(anim, Tiso);
                }
                if constexpr (GRAD) {
                    gfr = vfnma(gim, fTi, vmul(gre, fTr));
                    gfi = vfma(gim, fTr, vmul(gre, fTi));
                }
            }
            V Ure, Uim, gU, own[OWN ? 9 : 1];
            V zTr[INV && !INVC ? NZ : 1], zTi[INV && !INVC ? NZ : 1];
#pragma unroll
            for (int c = 0; c < NC; c++) {
                V cr[SLOTS];
                {
                    const PkV16<V> *src = reinterpret_cast<const PkV16<V> *>(cos_rec + c * SLOTS);
#pragma unroll
                    for (int q = 0; q < SLOTS * (int)sizeof(V) / 16; q++) {
                        const PkV16<V> t = src[q];
#pragma unroll
                        for (int i = 0; i < 16 / (int)sizeof(V); i++) cr[q * (16 / (int)sizeof(V)) + i] = t.v[i];
                    }
                }
                // ---- z = e^{i theta} T of the coset's operations
                V zr[CS], zi[CS];
                constexpr int NZC = INVC ? CS / 2 : CS;  // operations with phases of their own
                V m6[ANISO ? 6 : 1];
                if constexpr (ANISO) {
#pragma unroll
                    for (int q = 0; q < 6; q++) m6[q] = cr[HOFF + 3 + q];
                }
                if (!INV || INVC || c < NC / 2) {
#pragma unroll
                    for (int s = 0; s < NZC; s++) {
                        zr[s] = e_re[(c * CS + s) % NZ];
                        zi[s] = e_im[(c * CS + s) % NZ];
                    }
                    if constexpr (ANISO) {
                        // exponents: the diagonal and cross terms by character, one transform
                        V Q[CS], q[CS];
                        constexpr int kx = pk_char<CS, PAT>(3), ky = pk_char<CS, PAT>(5), kz = pk_char<CS, PAT>(6);
                        Q[0] = vfma(adp[2], m6[2], vfma(adp[1], m6[1], vmul(adp[0], m6[0])));
                        bool set[CS] = {true};
#pragma unroll
                        for (int j = 1; j < CS; j++) set[j] = false;
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            const int k = j == 0 ? kx : j == 1 ? ky : kz;
                            Q[k] = set[k] ? vfma(adp[3 + j], m6[3 + j], Q[k]) : vmul(adp[3 + j], m6[3 + j]);
                            set[k] = true;
                        }
#pragma unroll
                        for (int j = 1; j < CS; j++)
                            if (!set[j]) Q[j] = vdup<V>(R(0));
                        if constexpr (INVC && CS == 4) {
                            // an inversion leaves the exponent alone: two distinct ones
                            q[0] = vadd(Q[0], Q[1]);
                            q[1] = vsub(Q[0], Q[1]);
                        } else if constexpr (INVC) {
                            q[0] = Q[0];
                        } else {
                            pk_wht<CS>(Q, q);
                        }
#pragma unroll
                        for (int s = 0; s < NZC; s++) {
                            const V T = texp_v(q[s]);
                            zr[s] = vmul(zr[s], T);
                            zi[s] = vmul(zi[s], T);
                        }
                    }
                    if constexpr (INV && !INVC) {
#pragma unroll
                        for (int s = 0; s < CS; s++) {
                            zTr[(c * CS + s) % NZ] = zr[s];
                            zTi[(c * CS + s) % NZ] = zi[s];
                        }
                    }
                } else if constexpr (INV && !INVC) {
#pragma unroll
                    for (int s = 0; s < CS; s++) {
                        zr[s] = zTr[(c * CS + s) % NZ];
                        zi[s] = vneg(zTi[(c * CS + s) % NZ]);
                    }
                }
                // ---- sums over the coset by character: W (Re, Im) of u = f z, contracted with g
                V Gr[CS], Gi[CS];          // Re, Im of g W_k
                V Zr[CS], Zi[CS];          // transform of z (IAM, multipole adjoint, structure factors only)
                constexpr int HB = CS == 4 ? 2 : 1;  // INVC: the bit of the inversion's character
                if constexpr (IAM && INVC) {
                    // z of the images is the conjugate: the transform is real (even characters) or imaginary; half
                    // of it here, the factor 2 is in the weights (F) and at the final sums (derivatives)
                    V hr[CS / 2], hi[CS / 2], ar[CS / 2], ai[CS / 2];
#pragma unroll
                    for (int s = 0; s < CS / 2; s++) { ar[s] = zr[s]; ai[s] = zi[s]; }
                    pk_wht<CS / 2>(ar, hr);
                    pk_wht<CS / 2>(ai, hi);
#pragma unroll
                    for (int s = 0; s < CS / 2; s++) {
                        Zr[s] = hr[s];
                        Zi[s + CS / 2] = hi[s];
                    }
                    if (c == 0) { Ure = Zr[0]; Uim = vdup<V>(R(0)); }
                    if constexpr (GRAD) {
#pragma unroll
                        for (int k = 0; k < CS; k++) {
                            if (k & HB) {
                                Gr[k] = vneg(vmul(gfi, Zi[k]));
                                Gi[k] = vmul(gfr, Zi[k]);
                            } else {
                                Gr[k] = vmul(gfr, Zr[k]);
                                Gi[k] = vmul(gfi, Zr[k]);
                            }
                        }
                    }
                } else if constexpr (IAM) {
                    pk_wht<CS>(zr, Zr);
                    pk_wht<CS>(zi, Zi);
                    Ure = c == 0 ? Zr[0] : vadd(Ure, Zr[0]);
                    Uim = c == 0 ? Zi[0] : vadd(Uim, Zi[0]);
                    if constexpr (GRAD) {
#pragma unroll
                        for (int k = 0; k < CS; k++) {
                            Gr[k] = vfnma(gfi, Zi[k], vmul(gfr, Zr[k]));
                            Gi[k] = vfma(gfi, Zr[k], vmul(gfr, Zi[k]));
                        }
                    }
                } else {
                    V E[CS], O[CS], A[HC ? 5 : 1][CS];
                    V fr[CS], fi[CS];
                    if constexpr (HC) {
                        // angular sums by (l, character), then the radial weights
                        auto y = [&](int q) -> V { return cr[q]; };
                        auto p = [&](int q) -> V {
                            if constexpr (PG_SM) return sPg[q * TH + tid];
                            else return pg[q];
                        };
#pragma unroll
                        for (int q = 0; q < 9; q++) {
                            const int l = harmonic_l(q), k = pk_char<CS, PAT>(harmonic_class(q));
                            A[l][k] = slot_first<CS, PAT>(q) ? vmul(p(q), y(q)) : vfma(p(q), y(q), A[l][k]);
                        }
#pragma unroll
                        for (int k = 0; k < CS; k++) {
                            E[k] = k == 0 ? vfma(r[0], A[0][0], fs) : vdup<V>(R(0));
                            O[k] = k == 0 ? anim : vdup<V>(R(0));
                            if (slot_used<CS, PAT>(2, k)) E[k] = k == 0 ? vfma(r[2], A[2][k], E[k]) : vmul(r[2], A[2][k]);
                            if (slot_used<CS, PAT>(1, k)) O[k] = k == 0 ? vfma(r[1], A[1][k], O[k]) : vmul(r[1], A[1][k]);
                        }
                        if constexpr (HL) {
#pragma unroll
                            for (int q = 9; q < 25; q++) {
                                const int l = harmonic_l(q), k = pk_char<CS, PAT>(harmonic_class(q));
                                A[l][k] = slot_first<CS, PAT>(q) ? vmul(p(q), y(q)) : vfma(p(q), y(q), A[l][k]);
                            }
#pragma unroll
                            for (int k = 0; k < CS; k++) {
                                if (slot_used<CS, PAT>(4, k)) E[k] = vfma(r[4], A[4][k], E[k]);
                                if (slot_used<CS, PAT>(3, k)) O[k] = vfma(r[3], A[3][k], O[k]);
                            }
                        }
                        if constexpr (GRAD) {
                            pk_wht<CS>(E, fr);
                            pk_wht<CS>(O, fi);
                        }
                    } else {
                        // the table's value of every operation (excluded atoms: zero)
#pragma unroll
                        for (int s = 0; s < CS; s++) {
                            const int op = c * CS + s;
                            fr[s] = fi[s] = vdup<V>(R(0));
                            if constexpr (F64 && TABLE) {
                                if (active[0]) {
                                    const size_t a = (size_t)atom[0];
                                    const size_t col = a + (a >= (size_t)S.table_split ? S.table_shift : 0);
                                    const size_t ti = ((size_t)(h0 + hl) * S.table_stride + col) * NSC + op;
                                    if (S.table_d) {
                                        const double2 tv = S.table_d[ti];
                                        fr[s] = tv.x + anre;
                                        fi[s] = tv.y + anim;
                                    } else {
                                        const float2 tv = S.table_f[ti];
                                        fr[s] = widen(tv.x) + anre;
                                        fi[s] = widen(tv.y) + anim;
                                    }
                                }
                            }
                        }
                        if constexpr (INVC) {
#pragma unroll
                            for (int s = 0; s < CS / 2; s++) {
                                zr[s + CS / 2] = zr[s];
                                zi[s + CS / 2] = vneg(zi[s]);
                            }
                        }
                    }
                    if constexpr (MP || (HC && !GRAD)) {
                        pk_wht<CS>(zr, Zr);
                        pk_wht<CS>(zi, Zi);
                    }
                    if constexpr (HC && !GRAD) {
                        // U = sum_k (E_k + i O_k) Z_k
#pragma unroll
                        for (int k = 0; k < CS; k++) {
                            const bool first = c == 0 && k == 0;
                            Ure = first ? vmul(E[k], Zr[k]) : vfma(E[k], Zr[k], Ure);
                            Ure = vfnma(O[k], Zi[k], Ure);
                            if constexpr (!CEN) {
                                Uim = first ? vmul(E[k], Zi[k]) : vfma(E[k], Zi[k], Uim);
                                Uim = vfma(O[k], Zr[k], Uim);
                            }
                        }
                    } else {
                        V ur[CS], ui[CS];
#pragma unroll
                        for (int s = 0; s < CS; s++) {
                            ur[s] = vfnma(fi[s], zi[s], vmul(fr[s], zr[s]));
                            ui[s] = vfma(fi[s], zr[s], vmul(fr[s], zi[s]));
                        }
                        if constexpr (GRAD) {
                            V Wr[CS], Wi[CS];
                            pk_wht<CS>(ur, Wr);
                            pk_wht<CS>(ui, Wi);
                            Ure = c == 0 ? Wr[0] : vadd(Ure, Wr[0]);
                            Uim = c == 0 ? Wi[0] : vadd(Uim, Wi[0]);
#pragma unroll
                            for (int k = 0; k < CS; k++) {
                                Gr[k] = CEN ? vmul(gre, Wr[k]) : vfnma(gim, Wi[k], vmul(gre, Wr[k]));
                                Gi[k] = CEN ? vmul(gre, Wi[k]) : vfma(gim, Wr[k], vmul(gre, Wi[k]));
                            }
                        } else {
#pragma unroll
                            for (int s = 0; s < CS; s++) {
                                const bool first = c == 0 && s == 0;
                                Ure = first ? ur[s] : vadd(Ure, ur[s]);
                                Uim = first ? ui[s] : vadd(Uim, ui[s]);
                            }
                        }
                    }
                    if constexpr (MP) {
                        // adjoint weights by character: Re(g Z_k) for the even harmonics, Im(g Z_k) for the odd ones
                        V We[CS], Wo[CS];
#pragma unroll
                        for (int k = 0; k < CS; k++) {
                            We[k] = CEN ? vmul(gre, Zr[k]) : vfnma(gim, Zi[k], vmul(gre, Zr[k]));
                            Wo[k] = CEN ? vmul(gre, Zi[k]) : vfma(gim, Zr[k], vmul(gre, Zi[k]));
                        }
                        V dr[7];
#pragma unroll
                        for (int k = 0; k < NA; k++) {
                            const R *rm = reinterpret_cast<const R *>(st + SL.trm + toff[SAME ? 0 : k]) + 8 * hl;
#pragma unroll
                            for (int q = 0; q < 7; q++) vput(dr[q], k, rm[q]);
                        }
                        part[CH_PV] = vfma(dr[0], We[0], part[CH_PV]);
                        part[CH_KAPPA] = vfma(dr[1], We[0], part[CH_KAPPA]);
                        // kappa' and the populations: per (l, character) slot the weight r_l We (even l), -r_l Wo (odd l)
                        V kp;  // the reflection's kappa' sum apart: one rounding into the running sum
#pragma unroll
                        for (int l = 0; l < 5; l++) {
                            if (l >= NL) continue;
                            V QC[CS];
#pragma unroll
                            for (int k = 0; k < CS; k++) {
                                if (!slot_used<CS, PAT>(l, k)) continue;
                                const V Wk = (l & 1) ? Wo[k] : We[k];
                                const V t = vmul(A[l][k], Wk);
                                kp = l == 0 ? vmul(dr[2], t) : (l & 1) ? vfnma(dr[2 + l], t, kp) : vfma(dr[2 + l], t, kp);
                                QC[k] = vmul(r[l], Wk);
                            }
#pragma unroll
                            for (int q = l * l; q < (l + 1) * (l + 1); q++) {
                                const V Qk = QC[pk_char<CS, PAT>(harmonic_class(q))];
                                part[CH_PLM + q] = (l & 1) ? vfnma(Qk, cr[q], part[CH_PLM + q])
                                                           : vfma(Qk, cr[q], part[CH_PLM + q]);
                            }
                        }
                        part[CH_KAPPA_P] = vadd(part[CH_KAPPA_P], kp);
                    }
                }
                if constexpr (GRAD) {
                    // position and ADP adjoints: -h'_c Im(g W), -m6 Re(g W) of the class's character
                    gU = c == 0 ? Gr[0] : vadd(gU, Gr[0]);
                    if constexpr (OWN) {
                        if (c == 0) {
#pragma unroll
                            for (int q = 0; q < (ANISO ? 9 : 3); q++) own[q] = vdup<V>(R(0));
                        }
                    }
                    // channel q of xyz and (anisotropic) ADPs: the running sum, or the reflection's own
                    auto acc = [&](int q) -> V & {
                        if constexpr (OWN) return own[q];
                        else return part[q < 3 ? CH_XYZ + q : CH_ADP + q - 3];
                    };
#pragma unroll
                    for (int j = 0; j < 3; j++)
                        acc(j) = vfnma(cr[HOFF + j], Gi[pk_char<CS, PAT>(1 << j)], acc(j));
                    if constexpr (ANISO) {
#pragma unroll
                        for (int j = 0; j < 3; j++) acc(3 + j) = vfnma(m6[j], Gr[0], acc(3 + j));
#pragma unroll
                        for (int j = 3; j < 6; j++)
                            acc(3 + j) = vfnma(m6[j], Gr[pk_char<CS, PAT>(j == 3 ? 3 : j == 4 ? 5 : 6)], acc(3 + j));
                    }
                }
            }
            if constexpr (GRAD) {
                if constexpr (OWN) {
#pragma unroll
                    for (int q = 0; q < (ANISO ? 9 : 3); q++) {
                        V &p = part[q < 3 ? CH_XYZ + q : CH_ADP + q - 3];
                        p = vadd(p, own[q]);
                    }
                }
                part[CH_OCC] = vadd(part[CH_OCC], gU);
                if constexpr (!ANISO) part[CH_ADP] = vfnma(vdup<V>(sH2[hl]), gU, part[CH_ADP]);
            }
            if constexpr (IAM) {
                const V a = Ure;
                if constexpr (INVC) {
                    Ure = vmul(fTr, a);
                    Uim = vmul(fTi, a);
                } else {
                    Ure = vfnma(fTi, Uim, vmul(fTr, a));
                    Uim = vfma(fTr, Uim, vmul(fTi, a));
                }
            }
            const V wT = ANISO || IAM ? w : vmul(w, Tiso);
            fr_out = vsum(vmul(wT, Ure));
            if constexpr (CEN) fi_out = R(0);
            else fi_out = vsum(vmul(wT, Uim));
        };
        // a group's partial F over the lanes of the part, into sF
        auto reduce = [&](const PkEight<R> &F8, auto w32, const int g0, const int ng) {
            const R (&Fv)[8] = F8.v;
            const int wd = decltype(w32)::value ? decltype(w32)::value : width;
            const int o4 = wd >> 1, o3 = wd >> 2, o2 = wd >> 3;
            const bool b4 = lane & o4, b3 = lane & o3, b2 = lane & o2;
            if constexpr (CEN) {
                // four real values over the part's lanes: halves, quarters of them, then their sums
                R v2[2];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const R keep = b4 ? Fv[2 * q + 4] : Fv[2 * q], send = b4 ? Fv[2 * q] : Fv[2 * q + 4];
                    v2[q] = keep + shfl_xor<R>(send, o4);
                }
                R v1 = (b3 ? v2[1] : v2[0]) + shfl_xor<R>(b3 ? v2[0] : v2[1], o3);
                for (int o = o2; o > 0; o >>= 1) v1 += shfl_xor<R>(v1, o);
                const int idx = (b4 ? 2 : 0) + (b3 ? 1 : 0);
                if ((lane & (o3 - 1)) == 0 && idx < ng) sF[wrow * ht + g0 + idx] = R2{v1, R(0)};
                return;
            }
            // eight values over the part's lanes: halves, quarters, eighths of them, then their sums
            R v4[4], v2[2];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const R keep = b4 ? Fv[q + 4] : Fv[q], send = b4 ? Fv[q] : Fv[q + 4];
                v4[q] = keep + shfl_xor<R>(send, o4);
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const R keep = b3 ? v4[q + 2] : v4[q], send = b3 ? v4[q] : v4[q + 2];
                v2[q] = keep + shfl_xor<R>(send, o3);
            }
            R v1 = (b2 ? v2[1] : v2[0]) + shfl_xor<R>(b2 ? v2[0] : v2[1], o2);
            for (int o = o2 >> 1; o > 0; o >>= 1) v1 += shfl_xor<R>(v1, o);
            const int idx = (b4 ? 4 : 0) + (b3 ? 2 : 0) + (b2 ? 1 : 0);
            if ((lane & (o2 - 1)) == 0 && (idx >> 1) < ng) {
                R *dst = reinterpret_cast<R *>(&sF[wrow * ht + g0 + (idx >> 1)]);
                dst[idx & 1] = v1;
            }
        };
        // groups of four reflections: their eight sums over the warp by one butterfly reduce-scatter
        if (warp_any) {
#pragma unroll 1
            for (int g0 = seg0; g0 < seg0 + seg; g0 += 4) {
                const int ng = F64 ? min(4, seg) : 4;
                PkEight<R> Fv;
                // a group inside its lines runs as one straight stretch of code; one with a line start takes its
                // reflections in a loop (with large bodies every group does)
                bool straight = false;
                if constexpr (!ROLL_J) {
                    if (ng == 4) {
                    const int4 c4 = *reinterpret_cast<const int4 *>(sCont + g0);
                    straight = (c4.x & c4.y & c4.z & c4.w & (F64 ? 2 : 1)) != 0 && !(g0 == seg0 && fresh);
                    }
                }
                if (straight) {
                    if constexpr (!ROLL_J) {
#pragma unroll
                        for (int j = 0; j < 4; j++) reflection(g0 + j, PkNo{}, Fv.v[2 * j], Fv.v[2 * j + 1]);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 8; q++) Fv.v[q] = R(0);
#pragma unroll 1
                    for (int j = 0; j < ng; j++) {
                        R a, b;
                        reflection(g0 + j, PkYes{}, a, b);
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (q == j) { Fv.v[2 * q] = a; Fv.v[2 * q + 1] = b; }
                    }
                }
                // (whole warps in a copy of their own, with constant lane distances)
                if constexpr (!F64) {
                    reduce(Fv, PkInt<32>{}, g0, ng);
                } else {
                    if (width == 32) reduce(Fv, PkInt<32>{}, g0, ng);
                    else reduce(Fv, PkInt<0>{}, g0, ng);
                }
            }
        } else {
            for (int i = seg0 + lane % width; i < seg0 + seg; i += width) sF[wrow * ht + i] = R2{R(0), R(0)};
        }
        if (GRAD && ((k_sub + 1) % fold == 0 || h0 + ht >= h_end)) {
#pragma unroll
            for (int q = 0; q < NT; q++) {
                if (!ANISO && q > CH_ADP && q < CH_OCC) continue;
#pragma unroll
                for (int k = 0; k < NA; k++) {
                    const int col = q * kTileAtoms + k * TH + tid;
                    const R sum = sTot[col], yv = vget(part[q], k) - sCmp[col], tv = sum + yv;
                    sCmp[col] = (tv - sum) - yv;
                    sTot[col] = tv;
                }
                part[q] = vdup<V>(R(0));
            }
        }
        __syncthreads();
        for (int i = tid; i < ht; i += TH) {
            R sre = 0, sim = 0;  // over the warps of the part that took reflection i
            for (int wp = 0; wp < max(1, slots / 32); wp++) {
                const R2 v = sF[wp * ht + i];
                sre += v.x;
                sim += v.y;
            }
            const R two = IAM && INVC ? R(2) : R(1);
            atomicAdd(&C.f_acc[h0 + i].x, (double)(two * sre));
            if constexpr (!CEN) atomicAdd(&C.f_acc[h0 + i].y, (double)(two * sim));
        }
        __syncthreads();
    }
    if constexpr (GRAD) {
#pragma unroll
        for (int k = 0; k < NA; k++) {
            if (!active[k]) continue;
            double *G = C.g_acc + (size_t)atom[k] * kNch;
            auto total = [&](int q) {
                const int col = q * kTileAtoms + k * TH + tid;
                const double t = (double)sTot[col] - (double)sCmp[col];
                return IAM && INVC ? 2.0 * t : t;
            };
#pragma unroll
            for (int q = 0; q < NT; q++) {
                if (!ANISO && q > CH_ADP && q < CH_OCC) continue;
                atomicAdd(G + q, total(q));
            }
        }
    }
}

// a block's tile: the code of its ADP kind and of its angular sums (with or without l = 3, 4).  KIND 0, 1: the launch
// holds tiles without, with anisotropic ADPs only
template <typename V, int MODEL, bool MP, int NSC, int CS, bool GRAD, bool INV, int PAT, bool CEN, int KIND, bool ROLL>
__device__ __forceinline__ void pk_tile(const DevStructure &S, const CallBuffers &C, const PkLaunch &L, int tile,
                                        int chunk)
{
    const bool aniso = KIND == 1 || (KIND == 2 && tile >= L.T.n_plain);
    if constexpr (MODEL == MODEL_HC) {
        const int4 info = L.T.info[tile];
        if ((MP ? info.w : info.z) >= 3) {
            if (KIND != 0 && aniso) pk_body<V, MODEL, MP, KIND != 0, NSC, CS, GRAD, INV, PAT, CEN, ROLL, true>(S, C, L, tile, chunk);
            else pk_body<V, MODEL, MP, KIND == 1, NSC, CS, GRAD, INV, PAT, CEN, ROLL, true>(S, C, L, tile, chunk);
            return;
        }
    }
    if (KIND != 0 && aniso) pk_body<V, MODEL, MP, KIND != 0, NSC, CS, GRAD, INV, PAT, CEN, ROLL, false>(S, C, L, tile, chunk);
    else pk_body<V, MODEL, MP, KIND == 1, NSC, CS, GRAD, INV, PAT, CEN, ROLL, false>(S, C, L, tile, chunk);
}

// Blocks per SM that the register allocation aims at.  Two atoms per thread: six (168 registers, three warps per
// scheduler), but the compiler's choice (about 220, two warps) where the cap would spill: HC derivatives with cosets of
// four (5,000 isotropic atoms, P2_1 2_1 2_1: 1.48 ms without, 1.55 ms with the cap; 4,000 atoms, C2/c 1.11 and
// 1.03 ms).  One atom, FP32 without the multipole adjoint: four (128 registers; 96 and 168 within 4% of it).
template <typename V, int MODEL, bool MP, bool GRAD, int CS>
__host__ __device__ constexpr int pk_min_blocks()
{
    if (VTraits<V>::NA == 2) return MODEL == MODEL_HC && GRAD && CS == 4 ? 1 : 6;
    return sizeof(V) == 4 && !MP ? 4 : 1;
}

// one structure: block tile * n_chunks + reflection chunk, so that blocks that run together share a tile's code and types
// (one grid dimension: a structure has any number of tiles, the others hold 65,535).  KIND
// 2: both ADP kinds in one launch (FP64, and FP32 grids of a few blocks per SM, where a second launch costs more than
// it saves); 0, 1: one launch per kind (two kinds' code at once overflow the instruction caches)
template <typename V, int MODEL, bool MP, int NSC, int CS, bool GRAD, bool INV, int PAT, bool CEN, int KIND>
__global__ void __launch_bounds__(pk_threads<V>(), pk_min_blocks<V, MODEL, MP, GRAD, CS>())
pk_kernel(const __grid_constant__ DevStructure S, const __grid_constant__ CallBuffers C,
          const __grid_constant__ PkLaunch L)
{
    pk_tile<V, MODEL, MP, NSC, CS, GRAD, INV, PAT, CEN, KIND, KIND == 2>(
        S, C, L, blockIdx.x / L.n_chunks + (KIND == 1 ? L.T.n_plain : 0), blockIdx.x % L.n_chunks);
}

// many structures of one kernel form in one launch (kernel-parameter space holds up to kBatchItems): the block's item
// is the last with block_begin <= blockIdx.x
struct PkBatchItem {
    DevStructure S;
    CallBuffers C;
    PkLaunch L;
    int n_tiles;
};
struct PkBatch {
    int n;
    int block_begin[kBatchItems + 1];
    PkBatchItem item[kBatchItems];
};

template <typename V, int MODEL, int NSC, int CS, bool INV, int PAT, bool CEN>
__global__ void __launch_bounds__(pk_threads<V>(), pk_min_blocks<V, MODEL, false, true, CS>())
pk_batch_kernel(const __grid_constant__ PkBatch B)
{
    const int b = blockIdx.x;
    int lo = 0, hi = B.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (B.block_begin[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    const PkBatchItem &it = B.item[lo];
    const int lb = b - B.block_begin[lo], n_chunks = (B.block_begin[lo + 1] - B.block_begin[lo]) / it.n_tiles;
    pk_tile<V, MODEL, false, NSC, CS, true, INV, PAT, CEN, 2, true>(it.S, it.C, it.L, lb / n_chunks, lb % n_chunks);
}

}  // namespace dsf
