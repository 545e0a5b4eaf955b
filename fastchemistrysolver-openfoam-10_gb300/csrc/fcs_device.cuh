// fcs_device.cuh -- device building blocks of the per-cell stiff integrator.
//
// Execution model: a *cell group* of G threads (G = 32: one warp; G = 64..512:
// one thread block) owns one cell at a time and keeps the whole per-cell
// working set in a private slot of shared memory (or of global memory when it
// does not fit): the Jacobian / LU matrices, the stage vectors, the species
// and reaction scratch.  Threads own species rows i = rank (mod G).  All
// scalars that steer control flow (error norms, step sizes) come out of
// butterfly reductions, so every thread of a group holds bit-identical values
// and takes the same branches.
//
// Code size: on a full SM the warps are spread over all phases of a step and
// share one instruction cache.  A loop that strides by the group runs once or
// twice, so it is kept rolled (left alone, the compiler unrolls it by four);
// the solves of small groups load four columns ahead instead of eight, and the
// mixed kernel has one right-hand side for its FP32 and its FP64 attempts.  34
// species, Seulex, 64 threads, 4,560 cells: mixed 125 -> 98 ms, FP64 81 -> 72
// (of 26 cycles per instruction 11 had been spent waiting for it); 53 species,
// Rodas34 mixed 128 -> 110.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fcs_internal.h"
#include "../../include/fcs.h"

namespace fcs {

// ------------------------------------------------------------------------
// cell group

template<int G>
struct Grp {
    int rank;  // 0..G-1
    __device__ __forceinline__ void sync() const {
        if constexpr (G == 32) __syncwarp();
        else __syncthreads();
    }
};

// Sum over the group; every thread returns the same bits.
template<int G>
__device__ __forceinline__ double gsum(const Grp<G>& g, double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if constexpr (G == 32) {
        return v;
    } else {
        g.sync();
        if ((g.rank & 31) == 0) red[g.rank >> 5] = v;
        g.sync();
        double s = red[0];
#pragma unroll
        for (int w = 1; w < G / 32; w++) s += red[w];
        return s;
    }
}

// Two sums at once (fewer barriers).
template<int G>
__device__ __forceinline__ void gsum2(const Grp<G>& g, double& a, double& b, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if constexpr (G > 32) {
        g.sync();
        if ((g.rank & 31) == 0) { red[g.rank >> 5] = a; red[16 + (g.rank >> 5)] = b; }
        g.sync();
        double s = red[0], t = red[16];
#pragma unroll
        for (int w = 1; w < G / 32; w++) { s += red[w]; t += red[16 + w]; }
        a = s; b = t;
    }
}

// Bits of |v|, ordered as the magnitudes are, NaN above infinity.
__device__ __forceinline__ unsigned long long magnitude_bits(double v) {
    return static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffULL;
}

// Maximum over the group of magnitude bits (a NaN anywhere wins), as a double.
template<int G>
__device__ __forceinline__ double gmax_bits(const Grp<G>& g, unsigned long long v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long u = __shfl_xor_sync(0xffffffffu, v, o);
        v = u > v ? u : v;
    }
    if constexpr (G > 32) {
        unsigned long long* r = reinterpret_cast<unsigned long long*>(red);
        g.sync();
        if ((g.rank & 31) == 0) r[g.rank >> 5] = v;
        g.sync();
        v = r[0];
#pragma unroll
        for (int w = 1; w < G / 32; w++) v = r[w] > v ? r[w] : v;
    }
    return __longlong_as_double(static_cast<long long>(v));
}

// Two maxima at once of non-negative values (or NaN, which wins), compared
// as integers on their bit patterns: the order of non-negative doubles is the
// order of their bits, and NaN patterns sit above +inf.  No FP64 compares.
template<int G>
__device__ __forceinline__ void gmax2_nonneg(const Grp<G>& g, double& a, double& b, double* red) {
    unsigned long long x = static_cast<unsigned long long>(__double_as_longlong(a));
    unsigned long long y = static_cast<unsigned long long>(__double_as_longlong(b));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long u = __shfl_xor_sync(0xffffffffu, x, o);
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, y, o);
        x = u > x ? u : x;
        y = v > y ? v : y;
    }
    if constexpr (G > 32) {
        unsigned long long* r = reinterpret_cast<unsigned long long*>(red);
        g.sync();
        if ((g.rank & 31) == 0) { r[g.rank >> 5] = x; r[16 + (g.rank >> 5)] = y; }
        g.sync();
        x = r[0];
        y = r[16];
#pragma unroll
        for (int w = 1; w < G / 32; w++) {
            x = r[w] > x ? r[w] : x;
            y = r[16 + w] > y ? r[16 + w] : y;
        }
    }
    a = __longlong_as_double(static_cast<long long>(x));
    b = __longlong_as_double(static_cast<long long>(y));
}

// ------------------------------------------------------------------------
// Comparisons on the integer pipe.  An FP64 compare, minimum or maximum holds
// a scheduler as long as a multiply-add does (64 cycles); the order of
// doubles of one sign is the order of their bits, and NaN patterns sit above
// infinity.

__device__ __forceinline__ bool ordered(long long magnitude) { return magnitude <= 0x7ff0000000000000LL; }

// x > 0
__device__ __forceinline__ bool positive(double x) {
    const long long b = __double_as_longlong(x);
    return b > 0 && ordered(b);
}

// a < b for b >= 0 or NaN
__device__ __forceinline__ bool less_than(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    return x < y && ordered(y) && ordered(x & 0x7fffffffffffffffLL);
}

// max(|a|, |b|) as fmax takes it for b NaN
__device__ __forceinline__ double larger_magnitude(double a, double b) {
    return less_than(fabs(a), fabs(b)) ? fabs(b) : fabs(a);
}

// a <= b for b > 0 or NaN
__device__ __forceinline__ bool at_most(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    return x <= y && ordered(y) && ordered(x & 0x7fffffffffffffffLL);
}

// ------------------------------------------------------------------------
// slot layout (byte offsets inside one cell's workspace)

struct SlotLayout {
    int ld;            // matrix leading dimension (odd: conflict-free column walks)
    int offJ64, offLU64;  // FP64 views of the Jacobian / LU factors (LU64 == J64: in place)
    int offJ32, offLU32;  // FP32 views (mixed precision), inside the same matrix region
    int offVec;        // kNV vectors of n doubles
    int offVec32;      // 2 vectors of n floats (mixed-precision solves)
    int offSp;         // 7 species arrays (C, E, Einv, Cp, Ha, dBdT, dCpdT) [ns]
    int offInvD;       // [n] double
    int offScale;      // row / column equilibration factors [2n] double (mixed precision)
    int offPiv;        // [n] int
    int offRx;         // max(4 rc, values) doubles: the net rates, or one Jacobian chunk (fcs_lists.h)
    int rc;            // a quarter of the least doubles at offRx, in [1, nr]
    int offCur;        // [ns] ints, free
    int jv;            // Jacobian chunking (kJacChunk) the region at offRx holds
    int rw;            // threads that carry the partial sums of the group's reductions
    int offTb;         // M (third-body concentration), third-body column weight [nTB] each
    int offTable;      // Seulex extrapolation table [12][n] doubles
    int offRed;        // 48 doubles of reduction / broadcast scratch (32..36 thermo scalars, 37 log p, 38..39 LU, 38 step factor, 40 queue)
    int bytes;         // total, multiple of 16
};

constexpr int kNV = 12;  // stage / work vectors per slot

__host__ __device__ inline int align16(int x) { return (x + 15) & ~15; }

// Matrix region:
//   FP64 Rosenbrock : one FP64 matrix, factored in place
//   FP64 Seulex     : FP64 Jacobian + FP64 LU (the Jacobian is reused across orders)
//   mixed Rosenbrock: FP32 Jacobian + FP32 LU; the FP64 view (Jacobian assembly in
//                     FP64, and the FP64 fallback attempt) overlays both
//   mixed Seulex    : as FP64 Seulex, with the two FP32 matrices inside the FP64 Jacobian
// values: doubles wanted at offRx; rc: a quarter of the least there (clamped
// to [1, nr]).
__host__ __device__ inline SlotLayout make_layout(int ns, int nr, int nTB, bool mixed, bool seulex, int rc,
                                                  int values = 0) {
    SlotLayout L;
    const int n = ns + 1;
    L.ld = n | 1;
    const int m64 = align16(n * L.ld * 8), m32 = align16(n * L.ld * 4);
    int o = 0;
    L.offJ64 = 0;
    if (seulex) { L.offLU64 = m64; o = 2 * m64; }   // FP64 Jacobian (kept) + FP64 LU
    else if (mixed) { L.offLU64 = 0; o = m64 + m32; } // FP64 Jacobian (kept) + FP32 LU; FP64 fallback in place
    else { L.offLU64 = 0; o = m64; }                 // FP64 matrix factored in place
    L.offJ32 = 0;                                    // (unused: the Jacobian stays FP64)
    L.offLU32 = m64;                                 // after the FP64 Jacobian (inside LU64 for Seulex)
    L.offVec = o;   o = align16(o + kNV * n * 8);
    L.offVec32 = o; if (mixed) o = align16(o + 2 * n * 4);
    L.offSp = o;    o = align16(o + 7 * ns * 8);
    L.offInvD = o;  o = align16(o + n * 8);
    L.offScale = o; if (mixed) o = align16(o + 2 * n * 8);
    L.offPiv = o;   o = align16(o + n * 4);
    L.rc = rc < 1 ? 1 : (nr > 0 && rc > nr ? nr : rc);
    const int rx = 4 * L.rc > values ? 4 * L.rc : values;
    L.offRx = o;    o = align16(o + (rx * 8 > n * 4 ? rx * 8 : n * 4));  
    L.offCur = o;   o = align16(o + ns * 4);
    L.offTb = o;    o = align16(o + 2 * (nTB > 0 ? nTB : 1) * 8);
    L.offTable = o;
    if (seulex) o = align16(o + 12 * n * 8);
    L.offRed = o;   o = align16(o + 48 * 8);
    L.bytes = o;
    L.jv = 0;
    L.rw = 0;
    return L;
}

// What a cell's rates, right-hand side or time scale need: no matrix, two
// vectors, five species arrays, the net rates, M of the third bodies and the
// reduction scratch.  6 KB instead of 34 for 53 species, so that registers and
// not shared memory limit the cells of an SM.  The other offsets are not used.
inline SlotLayout make_source_layout(int ns, int nr, int nTB) {
    SlotLayout L{};
    const int n = ns + 1;
    int o = 0;
    L.offVec = o;   o = align16(o + 2 * n * 8);
    L.offSp = o;    o = align16(o + 5 * ns * 8);
    L.offRx = o;    o = align16(o + (nr > 0 ? nr : 1) * 8);
    L.offTb = o;    o = align16(o + (nTB > 0 ? nTB : 1) * 8);
    L.offRed = o;   o = align16(o + 48 * 8);
    L.bytes = o;
    return L;
}

// A Jacobian without the step around it: no stage vectors, pivots or scratch of
// the solves.  values: doubles of a chunk (or of the net rates).
inline SlotLayout make_jacobian_layout(int ns, int nTB, int values) {
    SlotLayout L{};
    const int n = ns + 1;
    L.ld = n | 1;
    int o = align16(n * L.ld * 8);
    L.offVec = o;   o = align16(o + 2 * n * 8);
    L.offSp = o;    o = align16(o + 7 * ns * 8);
    L.offRx = o;    o = align16(o + values * 8);
    L.offTb = o;    o = align16(o + 2 * (nTB > 0 ? nTB : 1) * 8);
    L.offRed = o;   o = align16(o + 48 * 8);
    L.bytes = o;
    return L;
}

template<class MT>
struct Slot {
    int ld, n, ns;
    MT* J;
    MT* LU;
    double* vec;      // vec + k*n is vector k
    float *x32, *r32; // FP32 solve vectors (mixed precision)
    double* J64;      // the FP64 Jacobian (== J for MT = double)
    double *C, *B, *Binv, *Cp, *Ha, *dBdT, *dCpdT;   // B = exp(-G/RT), Binv = 1/B
    double* invD;
    double *dr, *dc;
    int* piv;
    double* q;                     // net rates by packed reaction, or a Jacobian chunk's values
    int jv, rw;
    double *Mtb, *tbF;
    double* table;
    double* red;
    __device__ double* v(int k) const { return vec + k * n; }
};

template<class MT>
__device__ __forceinline__ Slot<MT> make_slot(char* base, const SlotLayout& L, const DevMech& M) {
    Slot<MT> s;
    s.ld = L.ld; s.n = M.n; s.ns = M.ns;
    if constexpr (sizeof(MT) == 8) {
        s.J = reinterpret_cast<MT*>(base + L.offJ64);
        s.LU = reinterpret_cast<MT*>(base + L.offLU64);
    } else {
        s.J = reinterpret_cast<MT*>(base + L.offJ32);
        s.LU = reinterpret_cast<MT*>(base + L.offLU32);
    }
    s.vec = reinterpret_cast<double*>(base + L.offVec);
    s.x32 = reinterpret_cast<float*>(base + L.offVec32);
    s.r32 = s.x32 + M.n;
    s.J64 = reinterpret_cast<double*>(base + L.offJ64);
    double* sp = reinterpret_cast<double*>(base + L.offSp);
    s.C = sp; s.B = sp + M.ns; s.Binv = sp + 2 * M.ns; s.Cp = sp + 3 * M.ns; s.Ha = sp + 4 * M.ns;
    s.dBdT = sp + 5 * M.ns; s.dCpdT = sp + 6 * M.ns;
    s.invD = reinterpret_cast<double*>(base + L.offInvD);
    s.dr = reinterpret_cast<double*>(base + L.offScale);
    s.dc = s.dr + M.n;
    s.piv = reinterpret_cast<int*>(base + L.offPiv);
    s.q = reinterpret_cast<double*>(base + L.offRx);
    s.jv = L.jv;
    s.rw = L.rw;
    double* tb = reinterpret_cast<double*>(base + L.offTb);
    const int nt = M.nTB > 0 ? M.nTB : 1;
    s.Mtb = tb; s.tbF = tb + nt;
    s.table = reinterpret_cast<double*>(base + L.offTable);
    s.red = reinterpret_cast<double*>(base + L.offRed);
    return s;
}

// ------------------------------------------------------------------------
// thermo (ThermoFunctionI.H)

__device__ __forceinline__ const double* species_coeffs(const DevMech& M, int i, double Tb) {
    // setPtrCoeffs (ThermoFunctionI.H:1-31)
    const double* base = M.coef + 32 * i;
    if (less_than(Tb, M.TcommonMin)) return base;
    if (less_than(M.TcommonMax, Tb)) return base + 16;
    return less_than(Tb, __ldg(&M.Tcommon[i])) ? base : base + 16;
}

// A species' NASA-7 set with the products of the coefficients and the
// polynomials' constants (formed on the host with the same rounding: eight
// FP64 instructions per species fewer in each evaluation).
struct Nasa { double a0, a1, a2, a3, a4, a5, a6, a1h, a2_6, a2_3, a3_12, a3_4, a4_20, a4_5; };

__device__ __forceinline__ Nasa load_nasa(const double* a) {
    Nasa c;
    c.a0 = __ldg(a + 0); c.a1 = __ldg(a + 1); c.a2 = __ldg(a + 2); c.a3 = __ldg(a + 3);
    c.a4 = __ldg(a + 4); c.a5 = __ldg(a + 5); c.a6 = __ldg(a + 6);
    c.a1h = __ldg(a + 7); c.a2_6 = __ldg(a + 8); c.a2_3 = __ldg(a + 9); c.a3_12 = __ldg(a + 10);
    c.a3_4 = __ldg(a + 11); c.a4_20 = __ldg(a + 12); c.a4_5 = __ldg(a + 13);
    return c;
}

// exponent of exp(-G/RT) (ThermoFunctionI.H:539-636)
__device__ __forceinline__ double gibbs_exponent(const Nasa& a, double T, double invT, double logT) {
    double v = fma(a.a4_20, T, a.a3_12);
    v = fma(v, T, a.a2_6);
    v = fma(v, T, a.a1h);
    v = fma(v, T, -(a.a5 * invT));
    v = v + a.a6;
    return fma(a.a0, logT - 1.0, v);
}

__device__ __forceinline__ double cp_of(const Nasa& a, double T, double RuInvW) {
    double v = fma(a.a4, T, a.a3);
    v = fma(v, T, a.a2);
    v = fma(v, T, a.a1);
    v = fma(v, T, a.a0);
    return RuInvW * v;
}

__device__ __forceinline__ double ha_of(const Nasa& a, double T, double RuInvW) {
    double v = fma(a.a4, T * 0.2, a.a3_4);
    v = fma(v, T, a.a2_3);
    v = fma(v, T, a.a1h);
    v = fma(v, T, a.a0);
    v = fma(v, T, a.a5);
    return RuInvW * v;
}

__device__ __forceinline__ double clampT(const DevMech& M, double T) {
    T = less_than(T, M.TlowMin) ? M.TlowMin : T;
    T = less_than(M.ThighMax, T) ? M.ThighMax : T;
    return T;
}

// ------------------------------------------------------------------------
// exp(x) in FP64 by Tang's table-driven method (P. T. P. Tang, "Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15(2):144-157, 1989), with 64 table entries:
//   x = (64 m + j) ln2/64 + r,  |r| <= ln2/128,
//   exp(x) = 2^m * 2^(j/64) * (1 + p(r)),  p(r) = r + r^2/2! + ... + r^5/5!
// (truncation below 4e-17).  N = 64 m + j is rounded with the 1.5*2^52
// shift, ln2/64 is split in a 36-bit head and a tail so N*head is exact, and
// 2^m is applied by adding m to the exponent field on the integer pipe.
// |x| > 707 (outside the range where 2^m stays a normal number) goes to the
// CUDA exp.  About 12 FP64 instructions.
__device__ const double kExp2Table[64] = {
    1.0, 1.0108892860517005, 1.0218971486541166, 1.0330248790212284,
    1.0442737824274138, 1.0556451783605572, 1.0671404006768237, 1.0787607977571199,
    1.0905077326652577, 1.102382583307841, 1.1143867425958924, 1.1265216186082418,
    1.1387886347566916, 1.1511892299529827, 1.1637248587775775, 1.1763969916502812,
    1.189207115002721, 1.202156731452703, 1.215247359980469, 1.22848053610687,
    1.241857812073484, 1.255380757024691, 1.2690509571917332, 1.2828700160787783,
    1.2968395546510096, 1.3109612115247644, 1.3252366431597413, 1.339667524053303,
    1.3542555469368927, 1.3690024229745905, 1.383909881963832, 1.3989796725383112,
    1.4142135623730951, 1.42961333839197, 1.4451808069770467, 1.460917794180647,
    1.4768261459394993, 1.4929077282912648, 1.5091644275934228, 1.5255981507445384,
    1.5422108254079407, 1.559004400237837, 1.5759808451078865, 1.593142151342267,
    1.6104903319492543, 1.6280274218573478, 1.645755478153965, 1.6636765803267364,
    1.681792830507429, 1.7001063537185235, 1.718619298122478, 1.7373338352737062,
    1.7562521603732995, 1.7753764925265212, 1.7947090750031072, 1.8142521755003989,
    1.8340080864093424, 1.8539791250833855, 1.8741676341103, 1.8945759815869656,
    1.9152065613971474, 1.9360617934922943, 1.9571441241754002, 1.978456026387951};

// Out of range arguments; one copy of the code (inlined, CUDA's exp stood in
// every rate expression, and the instruction cache is shared by all of them).
static __device__ __noinline__ double exp_out_of_range(double x) { return exp(x); }

__device__ __forceinline__ double fast_exp(double x) {
    // |x| <= 707 (0x4086180000000000), false for NaN
    if ((__double_as_longlong(x) & 0x7fffffffffffffffLL) > 0x4086180000000000LL) return exp_out_of_range(x);
    const double kInvL = 92.33248261689366;          // 64/ln2
    const double kL1 = 0.010830424696223417;         // head of ln2/64 (36 bits)
    const double kL2 = 2.572804622327669e-14;        // tail
    const double kShift = 6755399441055744.0;        // 1.5 * 2^52
    const double kk = fma(x, kInvL, kShift);
    const long long N = __double_as_longlong(kk) - 0x4338000000000000LL;
    const double Nf = kk - kShift;
    double r = fma(-Nf, kL1, x);
    r = fma(-Nf, kL2, r);
    double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
    q = fma(r, q, 1.0 / 6.0);
    q = fma(r, q, 0.5);
    q = fma(r, q, 1.0);
    const double p = r * q;
    const double S = __ldg(&kExp2Table[N & 63]);
    const double res = fma(S, p, S);
    return __longlong_as_double(__double_as_longlong(res) + ((N >> 6) << 52));
}

// OptReaction::fastPow (OptReaction.H:1405-1420)
__device__ __forceinline__ double fast_pow_int(double x, int order) {
    double xx = order < 0 ? 1 / x : x;
    double y = 1;
    for (int i = order; i != 0; i /= 2) {
        if (i % 2) y *= xx;
        xx *= xx;
    }
    return y;
}

// Pstd/(Ru T) and its inverse: the pressure factor of 1/Kc is (Pstd/(Ru T))^(-dnu)
struct PFactor { double P, invP; };

__device__ __forceinline__ PFactor pressure_factors(double Tc) {
    PFactor f;
    f.invP = kRu * Tc / kPstd;
    f.P = 1.0 / f.invP;
    return f;
}

constexpr double kInvKcClamp = 1.0 / kKcClamp;
constexpr double kInvKcClampG = 1.0 / kKcClampG;

// (Pstd/(Ru T))^(-dnu): the reference's table for |dnu| <= 2
// (ChemicalEquilibriumFunctionI.H:14-25), fastPow beyond it (RFG/JFG)
__device__ __forceinline__ double pressure_factor(const PFactor& pf, int dnu) {
    switch (dnu) {
        case -2: return pf.P * pf.P;
        case -1: return pf.P;
        case 1: return pf.invP;
        case 2: return pf.invP * pf.invP;
        default: return fast_pow_int(pf.invP, dnu);
    }
}

// The clamp of 1/Kc: RFG/JFG (more than 3 species on a side) use the other constant
template<class Rxn>
__device__ __forceinline__ double inv_kc_clamp(const Rxn& x) {
    return (x.nl > 3 || x.nr > 3) ? kInvKcClampG : kInvKcClamp;
}

// ------------------------------------------------------------------------
// rate constants

// PLOG: ln k linear in ln p between the bracketing rows, clamped to the end
// rows (ReactionRate.C:577-727, Jacobian.C:798-1000); returns k, sets dk/dT.
__device__ __forceinline__ double plog_rate(const DevMech& M, int ip, double p, double logP,
                                            double logT, double invT, double* dkdT) {
    const int o = __ldg(&M.plogOff[ip]);
    const int len = __ldg(&M.plogOff[ip + 1]) - o;
    const double* R = M.plogRow;
    double lk, dk;
    if (at_most(p, __ldg(&R[4 * o]))) {
        const double la = __ldg(&R[4 * o + 2]), b = __ldg(&R[4 * o + 3]), ta = __ldg(&M.plogTa[o]);
        lk = la + b * logT - ta * invT;
        dk = (b + ta * invT) * invT;
    } else if (at_most(__ldg(&R[4 * (o + len - 1)]), p)) {
        const int e = o + len - 1;
        const double la = __ldg(&R[4 * e + 2]), b = __ldg(&R[4 * e + 3]), ta = __ldg(&M.plogTa[e]);
        lk = la + b * logT - ta * invT;
        dk = (b + ta * invT) * invT;
    } else {
        int idx = 0;
        if (M.plogSorted) {
            // the first bracket that holds p: one below the number of rows
            // under p, counted without waiting for one load before the next
            #pragma unroll 4
            for (int j = 1; j < len - 1; j++) idx += less_than(__ldg(&R[4 * (o + j)]), p);
        } else for (int j = 0; j < len - 1; j++) {
            if (at_most(__ldg(&R[4 * (o + j)]), p) && at_most(p, __ldg(&R[4 * (o + j + 1)]))) { idx = j; break; }
        }
        const int a = o + idx, b = a + 1;
        const double lpa = __ldg(&R[4 * a + 1]), lpb = __ldg(&R[4 * b + 1]);
        const double laa = __ldg(&R[4 * a + 2]), lab = __ldg(&R[4 * b + 2]);
        const double ba = __ldg(&R[4 * a + 3]), bb = __ldg(&R[4 * b + 3]);
        const double ta = __ldg(&M.plogTa[a]), tb = __ldg(&M.plogTa[b]);
        const double fr = (logP - lpa) / (lpb - lpa);
        lk = laa + ba * logT - ta * invT + ((lab - laa) + (bb - ba) * logT - (tb - ta) * invT) * fr;
        dk = invT * (ba + ta * invT + (bb - ba + (tb - ta) * invT) * fr);
    }
    const double k = fast_exp(lk);
    *dkdT = k * dk;
    return k;
}

__device__ __forceinline__ RxnInfo load_rx(const RxnInfo* p) {
    // 64-byte record, four 16-byte loads through the read-only path
    RxnInfo x;
    const double2* s = reinterpret_cast<const double2*>(p);
    double2* d = reinterpret_cast<double2*>(&x);
    d[0] = __ldg(s);
    d[1] = __ldg(s + 1);
    d[2] = __ldg(s + 2);
    d[3] = __ldg(s + 3);
    return x;
}

// ------------------------------------------------------------------------
// fall-off reactions (ReactionRate.C:370-519, Jacobian.C:426-713,
// pressureReactionFunctionI.H): Kf = M K0 F / (1 + Pr), Pr = K0 M / kInf,
// F = 1 (Lindemann), Troe or SRI.  K0 is the reaction's own Arrhenius rate,
// kInf and the F parameters come from DevMech::fo; Tc is the clamped
// temperature.  With deriv, also dKf/dT and dKf/dM; the SRI branch uses dF/dT
// at fixed Pr, as the reference does (no dF/dPr dPr/dT term), the Troe branch
// the total derivative.

//
// Troe and SRI rates are chains of exponentials, logarithms and powers; a power
// alone holds a warp for some 5,800 cycles, and a group waits for the longest
// chain.  With W = 4, four neighbouring lanes evaluate one reaction (K0 is then
// formed here): each takes one of the exponentials, or every other logarithm or
// power, in the same instructions, and passes it on.  The arguments and so the
// results are those of W = 1.  16 species with 3 Troe and 3 SRI reactions: the
// rates of a right-hand side 35.4 -> 27.3 k cycles, 513 cells under Seulex 292 ->
// 271 ms.

struct FalloffK { double Kf, dKfdT, dKfdC; };

// The value of lane `of` of this lane's four
__device__ __forceinline__ double of_four(double v, int of) {
    const int lane = threadIdx.x & 31;
    return __shfl_sync(0xfu << (lane & ~3), v, (lane & ~3) + of);
}

template<int W>
static __device__ __noinline__ FalloffK falloff_rate(const DevMech& M, const RxnInfo& x, double K0, double dK0dT,
                                                     double Mt, double Tc, double logT, double invT, bool deriv) {
    const double* f = M.fo + (size_t)x.fo * 8;
    const double A2 = __ldg(f), b2 = __ldg(f + 1), Ta2 = __ldg(f + 2);
    const double argInf = fma(b2, logT, -(Ta2 * invT));
    const int sub = threadIdx.x & 3;
    double Kinf, e3 = 0, e4 = 0;  // e3, e4: the third and fourth exponential, W = 4
    if constexpr (W == 4) {
        double a3, a4;
        if (x.kind == FCS_RXN_TROE_FALLOFF) {
            a3 = -Tc * (1.0 / __ldg(f + 6));
            a4 = -__ldg(f + 5) * invT;
        } else {
            a3 = -__ldg(f + 4) * invT;
            a4 = -Tc * (1.0 / __ldg(f + 5));
        }
        const double a0 = x.tind ? 0.0 : fma(x.beta, logT, -(x.Ta * invT));
        const double e = fast_exp(sub == 0 ? a0 : sub == 1 ? argInf : sub == 2 ? a3 : a4);
        const double e0 = of_four(e, 0);
        Kinf = A2 * of_four(e, 1);
        e3 = of_four(e, 2);
        e4 = of_four(e, 3);
        K0 = x.tind ? x.A : x.A * e0;
        dK0dT = x.tind ? 0.0 : K0 * (fma(x.Ta, invT, x.beta) * invT);
    } else {
        Kinf = A2 * fast_exp(argInf);
    }
    const double dKinfdT = Kinf * (fma(Ta2, invT, b2) * invT);
    FalloffK o{0, 0, 0};
    if (W == 1 && x.kind == FCS_RXN_LINDEMANN_FALLOFF) {
        if (!deriv) {
            const double Pr = (K0 * Mt) / Kinf;
            o.Kf = Mt * (K0 / (Pr + 1.0));
            return o;
        }
        const double invKinf = 1.0 / Kinf;
        const double Pr = (K0 * Mt) * invKinf;
        const double dPrdT = fma(Mt, dK0dT, -(Pr * dKinfdT)) * invKinf;
        const double tmp = 1.0 / (1.0 + Pr);
        o.dKfdT = fma(tmp, Pr * dKinfdT, ((tmp * tmp) * dPrdT) * Kinf);
        o.dKfdC = (K0 * tmp) * tmp;
        o.Kf = Mt * (tmp * K0);
        return o;
    }
    const double small = 1e-15;
    const double Pr = K0 * Mt / Kinf;
    const double logTen = 2.302585092994045684;
    double logPr = 0;
    if (W == 1 || x.kind != FCS_RXN_TROE_FALLOFF) logPr = log10(fmax(Pr, small));
    double F, dFdT = 0, dFdPr = 0;
    if (x.kind == FCS_RXN_TROE_FALLOFF) {
        const double alpha = __ldg(f + 3), Ts = __ldg(f + 4), Tss = __ldg(f + 5), Tsss = __ldg(f + 6);
        const double invTsss = 1.0 / Tsss, invTs = 1.0 / Ts;
        const double eTsss = W == 4 ? e3 : fast_exp(-Tc * invTsss), eTss = W == 4 ? e4 : fast_exp(-Tss * invT);
        const double eTs = fast_exp(-Tc * invTs);
        const double Fcent = (1 - alpha) * eTsss + alpha * eTs + eTss;
        double logFcent;
        if constexpr (W == 4) {
            const double l = log10(fmax(sub & 1 ? Fcent : Pr, small));
            logPr = of_four(l, 0);
            logFcent = of_four(l, 1);
        } else {
            logFcent = log10(fmax(Fcent, small));
        }
        const double c = -0.4 - 0.67 * logFcent;
        const double n = 0.75 - 1.27 * logFcent;
        const double x1 = n - 0.14 * (logPr + c);
        const double invx1 = 1.0 / x1;
        const double x2 = (logPr + c) * invx1;
        const double x3 = 1 + (x2 * x2);
        const double invx3 = 1.0 / x3;
        const double x4 = logFcent * invx3;
        F = pow(10.0, x4);
        if (deriv) {
            const double dFcentdT = -(1 - alpha) * invTsss * eTsss - alpha * invTs * eTs + Tss * invT * invT * eTss;
            const double dlogFcentdT = Fcent >= small ? dFcentdT / Fcent / logTen : 0;
            const double dcdT = -0.67 * dlogFcentdT;
            const double dndT = -1.27 * dlogFcentdT;
            const double dx1dT = dndT - 0.14 * dcdT;
            const double dx2dT = (dcdT - x2 * dx1dT) * invx1;
            const double dx3dT = 2 * x2 * dx2dT;
            const double dx4dT = (dlogFcentdT - x4 * dx3dT) * invx3;
            const double dlogPrdPr = Pr >= small ? 1 / (logTen * Pr) : 0;
            const double dx1dPr = -0.14 * dlogPrdPr;
            const double dx2dPr = (dlogPrdPr - x2 * dx1dPr) * invx1;
            const double dx3dPr = 2 * x2 * dx2dPr;
            const double dx4dPr = -x4 * dx3dPr * invx3;
            dFdPr = logTen * F * dx4dPr;
            const double dPrdT = (Mt * dK0dT - Pr * dKinfdT) * (1.0 / Kinf);
            dFdT = logTen * F * dx4dT + dFdPr * dPrdT;
        }
    } else {
        const double a = __ldg(f + 3), b = __ldg(f + 4), c = __ldg(f + 5), d = __ldg(f + 6), e = __ldg(f + 7);
        const double X = 1 / (1 + (logPr * logPr));
        const double eb = W == 4 ? e3 : fast_exp(-b * invT), ec = W == 4 ? e4 : fast_exp(-Tc * (1.0 / c));
        const double psi = a * eb + ec;
        if constexpr (W == 4) {
            const double v = pow(sub & 1 ? Tc : psi, sub & 1 ? e : X);
            F = d * of_four(v, 0) * of_four(v, 1);
        } else {
            F = d * pow(psi, X) * pow(Tc, e);
        }
        if (deriv) {
            const double dpsidT = a * b / (Tc * Tc) * eb - 1 / c * ec;
            dFdT = F * (X / psi * dpsidT + e / Tc);
            const double dlogPrdPr = Pr >= small ? 1 / (logTen * Pr) : 0;
            const double dXdPr = -(X * X) * 2 * logPr * dlogPrdPr;
            dFdPr = F * log(psi) * dXdPr;
        }
    }
    const double invOnePlusPr = 1.0 / (1 + Pr);
    if (deriv) {
        const double dPrdT = (Mt * dK0dT - Pr * dKinfdT) * (1.0 / Kinf);
        o.dKfdT = F * invOnePlusPr * (Pr * dKinfdT) + F * invOnePlusPr * invOnePlusPr * dPrdT * Kinf +
                  K0 * invOnePlusPr * dFdT * Mt;
        o.dKfdC = K0 * invOnePlusPr * (F * invOnePlusPr + Pr * dFdPr);
    }
    o.Kf = Mt * (invOnePlusPr * F * K0);
    return o;
}

// Rates of one reaction of the special block: fall-off, non-equilibrium (the
// reverse rate its own Arrhenius, ReactionRate.C:362-367, 540-544) or
// third-body; Kf and Kr include M, and with deriv the temperature derivatives
// and dKf/dM, dKr/dM (Jacobian.C:401-422).
struct SpecialK { double Kf, dKfdT, dKfdC, Kr, dKrdT, dKrdC; };

// Mt: the reaction's third-body concentration (1 when it has none).  W = 4:
// four lanes to a Troe or SRI reaction (falloff_rate).
template<int W = 1>
static __device__ __forceinline__ SpecialK special_rates_m(const DevMech& M, const RxnInfo& x, const double Mt,
                                                        double Tc, double logT, double invT, bool deriv) {
    SpecialK o{0, 0, 0, 0, 0, 0};
    double K0 = x.A, dK0dT = 0;
    if (W == 1 && !x.tind) {
        K0 = x.A * fast_exp(fma(x.beta, logT, -(x.Ta * invT)));
        dK0dT = K0 * (fma(x.Ta, invT, x.beta) * invT);
    }
    if (x.fo >= 0) {
        const FalloffK k = falloff_rate<W>(M, x, K0, dK0dT, Mt, Tc, logT, invT, deriv);
        o.Kf = k.Kf;
        o.dKfdT = k.dKfdT;
        o.dKfdC = k.dKfdC;
    } else if (x.tb >= 0) {
        o.dKfdC = K0;
        o.Kf = K0 * Mt;
        o.dKfdT = dK0dT * Mt;
    } else {
        o.Kf = K0;
        o.dKfdT = dK0dT;
    }
    if (x.nq >= 0) {
        const double* f = M.fo + (size_t)x.nq * 8;
        const double Ar = __ldg(f), br = __ldg(f + 1), Tar = __ldg(f + 2);
        const double Kr = Ar * fast_exp(fma(br, logT, -(Tar * invT)));
        const double dKrdT = Kr * (fma(Tar, invT, br) * invT);
        if (x.tb >= 0) {
            o.dKrdC = Kr;
            o.Kr = Kr * Mt;
            o.dKrdT = dKrdT * Mt;
        } else {
            o.Kr = Kr;
            o.dKrdT = dKrdT;
        }
    }
    return o;
}

template<int W = 1>
static __device__ __forceinline__ SpecialK special_rates(const DevMech& M, const RxnInfo& x, const double* Mtb,
                                                      double Tc, double logT, double invT, bool deriv) {
    return special_rates_m<W>(M, x, x.tb >= 0 ? Mtb[x.tb] : 1.0, Tc, logT, invT, deriv);
}

// ------------------------------------------------------------------------
// Thermo scalars of one evaluation: log Tc, 1/Tc, num/p, Pstd/(Ru Tc) and its
// inverse.  A logarithm is 31 FP64 instructions and a division 8, and an
// instruction costs the same for one lane as for 32, so one warp takes the
// logarithm and another the divisions, side by side in its lanes, and a
// barrier (cheaper than one of those instructions) publishes them.

struct ThermoScalars { double logT, invT, numByP; PFactor pf; };

template<int G>
__device__ __forceinline__ ThermoScalars thermo_scalars(const Grp<G>& g, double* red, double Tc, double num, double p) {
    const int lane = g.rank & 31, warp = g.rank >> 5;
    ThermoScalars t;
    if (G == 32 || warp == 1) {
        const double q = (lane == 0 ? 1.0 : lane == 1 ? num : kRu * Tc) / (lane == 0 ? Tc : lane == 1 ? p : kPstd);
        const double inv = 1.0 / q;
        if constexpr (G == 32) {
            t.invT = __shfl_sync(0xffffffffu, q, 0);
            t.numByP = __shfl_sync(0xffffffffu, q, 1);
            t.pf.invP = __shfl_sync(0xffffffffu, q, 2);
            t.pf.P = __shfl_sync(0xffffffffu, inv, 2);
        } else {
            if (lane < 3) red[33 + lane] = q;
            if (lane == 2) red[36] = inv;
        }
    }
    if (G == 32 || warp == 0) {
        const double l = log(Tc);
        if constexpr (G == 32) t.logT = l;
        else if (lane == 0) red[32] = l;
    }
    if constexpr (G > 32) {
        g.sync();
        t.logT = red[32];
        t.invT = red[33];
        t.numByP = red[34];
        t.pf.invP = red[35];
        t.pf.P = red[36];
    }
    return t;
}

// Two sums sum_i a_i b_i in species order, as one thread would take them (a
// null: the constant ac): s.rw == 1, the lane mapping's sums.  The chains run
// in two lanes of one warp, so that the pair costs one FP64 instruction per
// species; the group's arrays are complete before (a barrier here).
struct SumOf { const double* a; double ac; const double* b; };
template<int G>
__device__ __forceinline__ void serial_sums(const Grp<G>& g, int n, const SumOf& f, const SumOf& h, double* red,
                                            double& x, double& y) {
    g.sync();
    if (g.rank < 2) {
        const SumOf s = g.rank ? h : f;
        double v = 0;
        #pragma unroll 8
        for (int i = 0; i < n; i++) v = fma(s.a ? s.a[i] : s.ac, s.b[i], v);
        red[g.rank] = v;
    }
    g.sync();
    x = red[0];
    y = red[1];
    if constexpr (G == 32) g.sync();
}

// M_t = sum_j eff[t][j] C_j (ThirdBodyFactor1D)
template<int G, class MT>
__device__ __forceinline__ void third_bodies(const Grp<G>& g, const DevMech& M, const Slot<MT>& s) {
    const int ns = M.ns;
    #pragma unroll 1
    for (int t = g.rank; t < M.nTB; t += G) {
        const double* e = M.eff + (size_t)t * ns;
        double m = 0;
        #pragma unroll 8
        for (int j = 0; j < ns; j++) m = fma(__ldg(&e[j]), s.C[j], m);
        s.Mtb[t] = m;
    }
}

// ------------------------------------------------------------------------
// reactions, one per thread, from the sorted records of fcs_lists.h

__device__ __forceinline__ RxnEv load_ev(const RxnEv* p) {
    RxnEv x;
    const double2* s = reinterpret_cast<const double2*>(p);
    double2* d = reinterpret_cast<double2*>(&x);
    d[0] = __ldg(s);
    d[1] = __ldg(s + 1);
    d[2] = __ldg(s + 2);
    d[3] = __ldg(s + 3);
    return x;
}

// The values of X at the first three slots of a side; unused slots hold
// species 0, so that the three loads go out together.
struct Three { double a, b, c; };
__device__ __forceinline__ Three load3(const double* X, const uint8_t* s) { return Three{X[s[0]], X[s[1]], X[s[2]]}; }
__device__ __forceinline__ double product3(const Three& t, int k) {
    double v = t.a;
    if (k > 1) v *= t.b;
    if (k > 2) v *= t.c;
    return v;
}
__device__ __forceinline__ bool three_at_most(const RxnEv& x) { return x.nl <= 3 && x.nr <= 3; }

__device__ __forceinline__ double product_over(const double* X, const uint8_t* s, int k) {
    double v = X[s[0]];
    #pragma unroll 1
    for (int q = 1; q < k; q++) v *= X[s[q]];
    return v;
}

// 1/Kc from per-species E = exp(-G/RT) and its inverse, no division:
// prod_reactants E prod_products 1/E (Pstd/(Ru T))^-dnu, with the reference's
// lower clamp of Kc (ReactionFunctionI.H:17; RFG's for more than 3 species on
// a side) as an upper clamp
__device__ __forceinline__ double inverse_kc(const RxnEv& x, const double* E, const double* Einv, const PFactor& pf) {
    double v;
    if (three_at_most(x)) {
        const Three e = load3(E, x.sl), i = load3(Einv, x.sr);
        v = product3(e, x.nl);
        v *= i.a;
        if (x.nr > 1) v *= i.b;
        if (x.nr > 2) v *= i.c;
    } else {
        v = product_over(E, x.sl, x.nl);
        #pragma unroll 1
        for (int q = 0; q < x.nr; q++) v *= Einv[x.sr[q]];
    }
    if (x.nr != x.nl) v *= pressure_factor(pf, x.nr - x.nl);
    const double cl = inv_kc_clamp(x);
    return less_than(cl, v) ? cl : v;
}

// Forward rate constant without third bodies; dkdT its temperature derivative
__device__ __forceinline__ double forward_k(const DevMech& M, const RxnEv& x, double p, double logP, double logT,
                                            double invT, double* dkdT) {
    if (x.plog >= 0) return plog_rate(M, x.plog, p, logP, logT, invT, dkdT);
    double Kf = x.A;
    *dkdT = 0;
    if (!x.tind) {
        Kf = x.A * fast_exp(fma(x.beta, logT, -(x.Ta * invT)));
        *dkdT = Kf * (fma(x.Ta, invT, x.beta) * invT);
    }
    return Kf;
}

template<class MT>
__device__ __forceinline__ double net_rate(const Slot<MT>& s, const RxnEv& x, double Kf, double Kr) {
    double CF, CR;
    if (three_at_most(x)) {
        const Three a = load3(s.C, x.sl), b = load3(s.C, x.sr);
        CF = product3(a, x.nl);
        CR = product3(b, x.nr);
    } else {
        CF = product_over(s.C, x.sl, x.nl);
        CR = product_over(s.C, x.sr, x.nr);
    }
    return Kf * CF - Kr * CR;
}

// The thread's rank when ranks are counted from warp w on
template<int G>
__device__ __forceinline__ int rank_from(const Grp<G>& g, int w) {
    return (g.rank + G - 32 * (w % (G / 32))) % G;
}

// Up to this many Troe (or SRI) rates are evaluated by four lanes each: one
// warp's worth, so that the warp still makes one pass over them (falloff_rate).
constexpr int kSpread = 8;

// Net rates of all reactions into s.q (ReactionRate.C:521-575 and the RF*
// functions), with the third-body concentrations.  The special block (first
// non-equilibrium to last fall-off reaction) runs in a loop of its own, so
// that the others carry neither the fall-off call nor a second Arrhenius: its
// Troe and SRI rates (some 300 FP64 instructions each) begin on a warp each,
// the other reactions on the warp after those (a warp further on, the last of
// them would wait behind the Troe rates: 271 -> 277 ms).  Without a special block the
// plain reactions do not wait for the third bodies.
template<int G, class MT>
__device__ __forceinline__ void net_rates(const Grp<G>& g, const DevMech& M, const Slot<MT>& s, double p, double logP,
                                          double Tc, const ThermoScalars& t) {
    third_bodies<G, MT>(g, M, s);
    const bool special = M.evSpecial < M.nr;
    if (special) {
        g.sync();
        #pragma unroll 1
        for (int part = 0; part < 3; part++) {
            const int k0 = part == 0 ? M.evTroe : part == 1 ? M.evSri : M.evSpecial;
            const int k1 = part == 0 ? M.evSri : part == 1 ? M.nr : M.evTroe;
            const bool spread = part < 2 && k1 - k0 <= kSpread;
            const int first = rank_from<G>(g, part);
            #pragma unroll 1
            for (int k = k0 + (spread ? first >> 2 : first); k < k1; k += G) {
                const RxnEv x = load_ev(M.ev + k);
                const RxnInfo xi = load_rx(M.rx + x.r);
                const SpecialK c = spread ? special_rates<4>(M, xi, s.Mtb, Tc, t.logT, t.invT, false)
                                          : special_rates(M, xi, s.Mtb, Tc, t.logT, t.invT, false);
                double Kr = c.Kr;  // non-equilibrium: its own reverse rate
                if (x.rev == 1) Kr = c.Kf * inverse_kc(x, s.B, s.Binv, t.pf);
                const double q = net_rate(s, x, c.Kf, Kr);
                if (!spread || (first & 3) == 0) s.q[x.r] = q;
            }
        }
    }
    #pragma unroll 1
    for (int part = 0; part < 2; part++) {
        const int end = part ? M.evSpecial : M.evThird;
        #pragma unroll 1
        for (int k = (part ? M.evThird : 0) + rank_from<G>(g, special ? 2 : 0); k < end; k += G) {
            const RxnEv x = load_ev(M.ev + k);
            double dk;
            double Kf = forward_k(M, x, p, logP, t.logT, t.invT, &dk);
            if (x.tb >= 0) Kf *= s.Mtb[x.tb];
            double Kr = 0;
            if (x.rev) Kr = Kf * inverse_kc(x, s.B, s.Binv, t.pf);
            s.q[x.r] = net_rate(s, x, Kf, Kr);
        }
        if (part == 0 && !special) g.sync();
    }
}

// v plus the terms of one lane's sum (n of them, of the group's most), in
// order; four terms' loads are issued together, lanes that are done add 0.
__device__ __forceinline__ double sum_terms(const uint32_t* __restrict__ con, int n, int most, const double* q,
                                            double v) {
    auto term = [&](uint32_t c, int k) {
        const long long b = __double_as_longlong(q[c >> 1]) ^ ((long long)(~c & 1u) << 63);
        return k < n ? __longlong_as_double(b) : 0.0;
    };
    int k = 0;
    #pragma unroll 1
    for (; k + 4 <= most; k += 4, con += 128) {
        const uint32_t c0 = __ldg(con), c1 = __ldg(con + 32), c2 = __ldg(con + 64), c3 = __ldg(con + 96);
        const double a = term(c0, k), b = term(c1, k + 1), c = term(c2, k + 2), d = term(c3, k + 3);
        v += a;
        v += b;
        v += c;
        v += d;
    }
    #pragma unroll 1
    for (; k < most; k++, con += 32) v += term(__ldg(con), k);
    return v;
}

// out[i] = net molar production of species i over s.q, in reaction order
template<int G, class MT>
__device__ __forceinline__ void net_production(const Grp<G>& g, const DevMech& M, const Slot<MT>& s, double* out) {
    const int lane = g.rank & 31;
    #pragma unroll 1
    for (int k = g.rank >> 5; k < M.prod.groups; k += G / 32) {
        const uint32_t e = __ldg(M.prod.elem + 32 * k + lane);
        int n = e & 0xffff;
        if (n == kLongSum) n = __ldg(M.prod.len + 32 * k + lane);
        const int most = __shfl_sync(0xffffffffu, n, 0), i = e >> 16;
        const double v = sum_terms(M.prod.con + __ldg(M.prod.off + k) + lane, n, most, s.q, 0.0);
        if (i != 0xffff) out[i] = v;
    }
}

// ------------------------------------------------------------------------
// right-hand side: FastChemistryModel::derivatives (FastChemistryModel.C:194-273
// for mode 1, 340-417 for mode 2) over OptReaction::dNdtByV
// (ReactionRate.C:732-1503).  YT is clamped (Y >= 0) in place.
//
// Bound by the count of FP64 warp instructions (19 cycles each per SM) when
// the SM is full of cells and by their latency when it holds one.  Reactions
// sorted by path, sums by length, scalars side by side, compares on integers:
// 877 -> 723 instructions on 53 species with 64 threads, fcs_rhs on
// 2,001 cells 0.19 -> 0.15 ms.

template<int G, class MT>
__device__ __noinline__ void rhs_eval(const Grp<G>& g, const DevMech& M, const Slot<MT>& s, double p,
                         double* YT, double* out, int mode) {
    const int ns = M.ns;
    const int r0 = g.rank < s.rw ? g.rank : ns;  // the threads that carry the partial sums
    const double T = YT[ns];
    const double Tc = clampT(M, T);
    const ThermoScalars t = thermo_scalars(g, s.red, Tc, kRu * T, p);
    double invrhoM = 0;
    if (s.rw == 1) {
        #pragma unroll 1
        for (int i = g.rank; i < ns; i += G) {
            const double y0 = YT[i];
            s.C[i] = (positive(y0) ? y0 : 0.0) * __ldg(&M.invW[i]);
        }
        const SumOf f{nullptr, t.numByP, s.C};
        double same;
        serial_sums(g, ns, f, f, s.red, invrhoM, same);
    } else {
        #pragma unroll 1
        for (int i = r0; i < ns; i += s.rw) {
            const double y0 = YT[i];
            invrhoM = fma((positive(y0) ? y0 : 0.0) * __ldg(&M.invW[i]), t.numByP, invrhoM);
        }
        invrhoM = gsum(g, invrhoM, s.red);
    }
    const double rhoM = 1.0 / invrhoM;
    const double Tp = mode == 2 ? T : Tc;
    #pragma unroll 1
    for (int i = g.rank; i < ns; i += G) {
        const double invW = __ldg(&M.invW[i]);
        const double y0 = YT[i], y = positive(y0) ? y0 : 0.0;
        YT[i] = y;
        s.C[i] = rhoM * invW * y;
        const Nasa a = load_nasa(species_coeffs(M, i, Tc));
        const double Ei = fast_exp(gibbs_exponent(a, Tc, t.invT, t.logT));
        s.B[i] = Ei;
        s.Binv[i] = 1.0 / Ei;
        const double RuInvW = __ldg(&M.RuInvW[i]);
        s.Cp[i] = cp_of(a, Tp, RuInvW);
        s.Ha[i] = ha_of(a, Tp, RuInvW);
    }
    g.sync();
    net_rates<G, MT>(g, M, s, p, s.red[37], Tc, t);
    g.sync();
    net_production<G, MT>(g, M, s, out);
    g.sync();
    #pragma unroll 1
    for (int i = g.rank; i < ns; i += G) out[i] = (__ldg(&M.W[i]) * invrhoM) * out[i];
    double cpm = 0, dtd = 0;
    if (s.rw == 1) {
        serial_sums(g, ns, SumOf{YT, 0, s.Cp}, SumOf{s.Ha, 0, out}, s.red, cpm, dtd);
    } else {
        if (s.rw < G) g.sync();
        #pragma unroll 1
        for (int i = r0; i < ns; i += s.rw) {
            cpm = fma(YT[i], s.Cp[i], cpm);
            dtd = fma(s.Ha[i], out[i], dtd);
        }
        gsum2(g, cpm, dtd, s.red);
    }
    if (g.rank == 0) out[ns] = -dtd / cpm;
    g.sync();
}

// ------------------------------------------------------------------------
// FastChemistryModel::tc (FastChemistryModel.C:589-651) over OptReaction::Tc
// (Tc.C:3-834): c = rho Y / W (not clamped); per reaction the forward and
// reverse molar rates summed over the products / reactants,
// wf = n_products Kf CF and wr = n_reactants Kr CR, with Kc from the ratio of
// Gibbs exponentials times fastPow(Pstd/(Ru T), dnu) clamped at
// 1.49011611938476e-8; tc = sum(w) / sum(w^2) * sum(c).  Returns tc to every
// thread.

// 1/Kc of a reaction whose factors leave the range of doubles (inf, or NaN from
// inf times 0): the quotient factor by factor; NaN ends on the clamp.
static __device__ __noinline__ double inverse_kc_by_division(const RxnEv& x, const double* E, const PFactor& pf) {
    double Kc = 1.0;
    #pragma unroll 1
    for (int q = 0; q < x.nl; q++) Kc = Kc / E[x.sl[q]];
    #pragma unroll 1
    for (int q = 0; q < x.nr; q++) Kc = Kc * E[x.sr[q]];
    Kc *= fast_pow_int(pf.P, x.nr - x.nl);
    return 1.0 / (Kc > kKcClampG ? Kc : kKcClampG);
}

template<int G, class MT>
__device__ __noinline__ double tc_eval(const Grp<G>& g, const DevMech& M, const Slot<MT>& s, double p, double T,
                                       double rho, const double* Y) {
    const int ns = M.ns;
    const double Tc = clampT(M, T);
    const ThermoScalars t = thermo_scalars(g, s.red, Tc, kRu * T, p);
    double sumc = 0;
    #pragma unroll 1
    for (int i = g.rank; i < ns; i += G) {
        const double ci = rho * Y[i] / __ldg(&M.W[i]);
        s.C[i] = ci;
        sumc += ci;
        const Nasa a = load_nasa(species_coeffs(M, i, Tc));
        const double E = fast_exp(gibbs_exponent(a, Tc, t.invT, t.logT));
        s.B[i] = E;
        s.Binv[i] = 1.0 / E;
    }
    sumc = gsum(g, sumc, s.red);
    g.sync();
    third_bodies<G, MT>(g, M, s);
    const double logP = s.red[37];
    double sw = 0, sw2 = 0;
    // Tc.C:578-600: the reverse rate only through Kc (1/Kc from the species'
    // factors, clamped at 1/1.49011611938476e-8 for every kind here); a
    // non-equilibrium reaction counts with its forward rate alone
    auto finish = [&](const RxnEv& x, const double Kf) {
        double Kr = 0;
        if (x.rev == 1) {
            double v = product_over(s.B, x.sl, x.nl);
            #pragma unroll 1
            for (int q = 0; q < x.nr; q++) v *= s.Binv[x.sr[q]];
            if (x.nr != x.nl) v *= pressure_factor(t.pf, x.nr - x.nl);
            // v > clamp on the integer pipe; v is a product of positive factors or NaN
            const unsigned long long bits = __double_as_longlong(v);
            if (bits > (unsigned long long)__double_as_longlong(kInvKcClampG))
                v = bits < 0x7ff0000000000000ULL ? kInvKcClampG : inverse_kc_by_division(x, s.B, t.pf);
            Kr = Kf * v;
        }
        double CF, CR;
        if (three_at_most(x)) {
            CF = product3(load3(s.C, x.sl), x.nl);
            CR = product3(load3(s.C, x.sr), x.nr);
        } else {
            CF = product_over(s.C, x.sl, x.nl);
            CR = product_over(s.C, x.sr, x.nr);
        }
        const double wf = x.nr * (Kf * CF), wr = x.nl * (Kr * CR);
        sw += wf + wr;
        sw2 = fma(wf, wf, fma(wr, wr, sw2));
    };
    #pragma unroll 1
    for (int part = 0; part < 2; part++) {
        const int end = part ? M.evSpecial : M.evThird;
        #pragma unroll 1
        for (int k = (part ? M.evThird : 0) + g.rank; k < end; k += G) {
            const RxnEv x = load_ev(M.ev + k);
            double dk;
            double Kf = forward_k(M, x, p, logP, t.logT, t.invT, &dk);
            if (x.tb >= 0) Kf *= s.Mtb[x.tb];
            finish(x, Kf);
        }
        if (part == 0) g.sync();
    }
    #pragma unroll 1
    for (int k = M.evSpecial + g.rank; k < M.nr; k += G) {
        const RxnEv x = load_ev(M.ev + k);
        const RxnInfo xi = load_rx(M.rx + x.r);
        finish(x, special_rates(M, xi, s.Mtb, Tc, t.logT, t.invT, false).Kf);
    }
    gsum2(g, sw, sw2, s.red);
    return sw2 == 0 ? 1e300 : sw / sw2 * sumc;
}

// ------------------------------------------------------------------------
// FastChemistryModel::calculate (FastChemistryModel.C:715-755): concentrations
// from the given density without clamping, RR_i = dNdtByV_i W_i.  Returns
// -sum Hf_i RR_i (Qdot, FastChemistryModel.C:656-685) to every thread.

template<int G, class MT>
__device__ __noinline__ double rates_eval(const Grp<G>& g, const DevMech& M, const Slot<MT>& s,
                                          double p, double T, double rho, const double* Y, double* RR) {
    const int ns = M.ns;
    const double Tc = clampT(M, T);
    const ThermoScalars t = thermo_scalars(g, s.red, Tc, kRu * Tc, p);
    #pragma unroll 1
    for (int i = g.rank; i < ns; i += G) {
        s.C[i] = rho * Y[i] / __ldg(&M.W[i]);
        const Nasa a = load_nasa(species_coeffs(M, i, Tc));
        const double Ei = fast_exp(gibbs_exponent(a, Tc, t.invT, t.logT));
        s.B[i] = Ei;
        s.Binv[i] = 1.0 / Ei;
    }
    g.sync();
    net_rates<G, MT>(g, M, s, p, s.red[37], Tc, t);
    g.sync();
    net_production<G, MT>(g, M, s, RR);
    g.sync();
    #pragma unroll 1
    for (int i = g.rank; i < ns; i += G) RR[i] = RR[i] * __ldg(&M.W[i]);
    if (s.rw < G) g.sync();
    double qd = 0;
    #pragma unroll 1
    for (int i = g.rank < s.rw ? g.rank : ns; i < ns; i += s.rw) qd -= __ldg(&M.hf[i]) * RR[i];
    qd = gsum(g, qd, s.red);
    g.sync();
    return qd;
}

// ------------------------------------------------------------------------
// analytic Jacobian: FastChemistryModel::jacobian (FastChemistryModel.C:489-572)
// over OptReaction::ddNdtByVdcTp (Jacobian.C:5-1004, JF11..JF33) and the dC/dY
// conversion (Jacobian.C:2814-2858 exact written as diagonal scaling plus a
// rank-1 correction, 4541-4568 fast, 3709-3741 T column, 3743-3793 T row).
// Writes J (row-major, leading dimension s.ld) and f = dy/dt; YT clamped in
// place.  With iterate, J receives the iteration matrix shift I - J instead.
//
// One thread evaluates a reaction with all its d q / d C; then every element
// of the matrix that any reaction touches is one sum, as are the species'
// net production (collected in the temperature row) and dq/dT (in the
// temperature column).  The former column owners walked incidence lists of
// unequal length in which reactants and products took different branches:
// 3,011 FP64 warp instructions on 53 species with 64 threads, now 2,043, and
// 2,000 such matrices 0.65 -> 0.50 ms.

// d q / d C of every occurrence of x's species, into v (reactants, then
// products when there is a reverse rate): the rate constant times the side's
// other concentrations (the first slot of the same species left out)
__device__ __forceinline__ void rate_gradients(const RxnEv& x, const double* C, double Kf, double Kr, double* v) {
    if (three_at_most(x)) {
        auto side = [&](const Three& c, int k, unsigned f1, unsigned f2, double K, double* o) {
            double d = K;
            if (k > 1) d *= c.b;
            if (k > 2) d *= c.c;
            o[0] = d;
            if (k > 1) {
                d = K * (f1 ? c.a : c.b);
                if (k > 2) d *= c.c;
                o[1] = d;
            }
            if (k > 2) o[2] = K * (f2 == 0 ? c.b : c.a) * (f2 == 2 ? c.b : c.c);
        };
        side(load3(C, x.sl), x.nl, x.first >> 2 & 3, x.first >> 4 & 3, Kf, v);
        if (x.rev) side(load3(C, x.sr), x.nr, x.first >> 11 & 7, x.first >> 14 & 7, -Kr, v + x.nl);
        return;
    }
    #pragma unroll 1
    for (int a = 0; a < x.nl; a++) {
        const int skip = x.first >> (2 * a) & 3;
        double d = Kf;
        #pragma unroll 1
        for (int q = 0; q < x.nl; q++)
            if (q != skip) d *= C[x.sl[q]];
        v[a] = d;
    }
    if (!x.rev) return;
    #pragma unroll 1
    for (int a = 0; a < x.nr; a++) {
        const int skip = x.first >> (8 + 3 * a) & 7;
        double d = -Kr;
        #pragma unroll 1
        for (int q = 0; q < x.nr; q++)
            if (q != skip) d *= C[x.sr[q]];
        v[x.nl + a] = d;
    }
}

template<int G, class MT>
__device__ __noinline__ void jac_eval(const Grp<G>& g, const DevMech& M, const Slot<MT>& s, double p,
                         double* YT, double* f, MT* J, int fast, bool iterate, double shift) {
    const int ns = M.ns, n = M.n, ld = s.ld;
    const int r0 = g.rank < s.rw ? g.rank : ns;
    const double T = YT[ns];
    const double Tc = clampT(M, T);
    // JacobianThermo (ThermoFunctionI.H:33-371) at the clamped temperature
    const ThermoScalars t = thermo_scalars(g, s.red, Tc, kRu * Tc, p);
    const double logT = t.logT, invT = t.invT;
    double rs = 0, mws = 0;
    if (s.rw == 1) {
        #pragma unroll 1
        for (int i = g.rank; i < ns; i += G) {
            const double y0 = YT[i], y = positive(y0) ? y0 : 0.0;
            YT[i] = y;
            s.C[i] = y * __ldg(&M.invW[i]);
        }
        serial_sums(g, ns, SumOf{nullptr, t.numByP, s.C}, SumOf{YT, 0, M.invW}, s.red, rs, mws);
    } else {
        #pragma unroll 1
        for (int i = r0; i < ns; i += s.rw) {
            const double y0 = YT[i], y = positive(y0) ? y0 : 0.0, invW = __ldg(&M.invW[i]);
            rs = fma(t.numByP, y * invW, rs);
            mws = fma(y, invW, mws);
        }
        gsum2(g, rs, mws, s.red);
    }
    const double rhoM = 1.0 / rs, invRhoM = rs, MW = 1.0 / mws;
    #pragma unroll 1
    for (int i = g.rank; i < ns; i += G) {
        const double y0 = YT[i], y = positive(y0) ? y0 : 0.0, invW = __ldg(&M.invW[i]);
        YT[i] = y;
        const Nasa a = load_nasa(species_coeffs(M, i, Tc));
        s.C[i] = rhoM * y * invW;
        const double Ei = fast_exp(gibbs_exponent(a, Tc, invT, logT));
        s.B[i] = Ei;
        s.Binv[i] = 1.0 / Ei;
        s.dBdT[i] = fma(fma(a.a5, invT, a.a0), invT,
                        fma(fma(fma(a.a4_5, Tc, a.a3_4), Tc, a.a2_3), Tc, a.a1h));
        const double RuInvW = __ldg(&M.RuInvW[i]);
        s.Cp[i] = cp_of(a, Tc, RuInvW);
        s.dCpdT[i] = RuInvW * fma(Tc, fma(Tc, fma(Tc, 4 * a.a4, 3 * a.a3), 2 * a.a2), a.a1);
        s.Ha[i] = ha_of(a, Tc, RuInvW);
    }
    for (int idx = g.rank; idx < n * ld; idx += G) J[idx] = MT(0);
    g.sync();
    third_bodies<G, MT>(g, M, s);
    if constexpr (G == 32) g.sync();
    double cpm = 0, dcpm = 0;  // the sums' barriers publish the third bodies
    if (s.rw == 1) {
        serial_sums(g, ns, SumOf{YT, 0, s.Cp}, SumOf{YT, 0, s.dCpdT}, s.red, cpm, dcpm);
    } else {
        #pragma unroll 1
        for (int i = r0; i < ns; i += s.rw) {
            cpm = fma(YT[i], s.Cp[i], cpm);
            dcpm = fma(YT[i], s.dCpdT[i], dcpm);
        }
        gsum2(g, cpm, dcpm, s.red);
    }
    const double CpM = cpm, dCpMdT = dcpm;
    const double logP = s.red[37];
    const JacLists& L = M.jac[s.jv];
    const int size = L.size;
    // Kr, dKr/dT and dKr/dM through Kc (JF* reversible branch)
    auto through_kc = [&](const RxnEv& x, const double Kf, const double dKfdT, const double dKfdC,
                          double& Kr, double& dKrdT, double& dKrdC) {
        const double invKc = inverse_kc(x, s.B, s.Binv, t.pf);
        double sv, sl;
        if (three_at_most(x)) {
            const Three v = load3(s.dBdT, x.sr), l = load3(s.dBdT, x.sl);
            sv = v.a;
            if (x.nr > 1) sv += v.b;
            if (x.nr > 2) sv += v.c;
            sl = l.a;
            if (x.nl > 1) sl += l.b;
            if (x.nl > 2) sl += l.c;
        } else {
            sv = s.dBdT[x.sr[0]];
            #pragma unroll 1
            for (int q = 1; q < x.nr; q++) sv += s.dBdT[x.sr[q]];
            sl = s.dBdT[x.sl[0]];
            #pragma unroll 1
            for (int q = 1; q < x.nl; q++) sl += s.dBdT[x.sl[q]];
        }
        const double dKcdTByKc = (sv - sl) - (x.nr - x.nl) * invT;
        Kr = Kf * invKc;
        // the Kc term of dKr/dT is dropped when Kc sits on its clamp (JacobianFunctionI.H:246-249)
        dKrdT = dKfdT * invKc - (less_than(invKc, inv_kc_clamp(x)) ? Kr * dKcdTByKc : 0.0);
        dKrdC = dKfdC * invKc;
    };
    auto finish = [&](const RxnEv& x, int l, const double Kf, const double dKfdT, const double dKfdC,
                      const double Kr, const double dKrdT, const double dKrdC) {
        double CF, CR;
        if (three_at_most(x)) {
            CF = product3(load3(s.C, x.sl), x.nl);
            CR = product3(load3(s.C, x.sr), x.nr);
        } else {
            CF = product_over(s.C, x.sl, x.nl);
            CR = product_over(s.C, x.sr, x.nr);
        }
        s.q[l] = Kf * CF - Kr * CR;
        s.q[size + l] = dKfdT * CF - dKrdT * CR;
        // third-body weight w = dKf/dM CF - dKr/dM CR
        if (x.tb >= 0) s.tbF[x.tb] = dKfdC * CF - dKrdC * CR;
        rate_gradients(x, s.C, Kf, Kr, s.q + x.ent);
    };
    #pragma unroll 1
    for (int c = 0, c0 = 0; c0 < M.nr; c++, c0 += size) {
        const int c1 = min(M.nr, c0 + size);
        const int special = __ldg(&L.chunk[c].special);
        #pragma unroll 1
        for (int k = c0 + rank_from<G>(g, special < c1 ? 2 : 0); k < special; k += G) {
            const RxnEv x = load_ev(L.ev + k);
            double dKfdT;
            double Kf = forward_k(M, x, p, logP, logT, invT, &dKfdT);
            double dKfdC = 0;
            if (x.tb >= 0) {
                const double Mt = s.Mtb[x.tb];
                dKfdC = Kf;
                Kf *= Mt;
                dKfdT *= Mt;
            }
            double Kr = 0, dKrdT = 0, dKrdC = 0;
            if (x.rev) through_kc(x, Kf, dKfdT, dKfdC, Kr, dKrdT, dKrdC);
            finish(x, x.r - c0, Kf, dKfdT, dKfdC, Kr, dKrdT, dKrdC);
        }
        const int troe = __ldg(&L.chunk[c].troe), sri = __ldg(&L.chunk[c].sri);
        #pragma unroll 1
        for (int part = 0; part < 3; part++) {
            // Troe rates start at warp 0, SRI rates at warp 1, the others at warp 2
            const int k0 = part == 0 ? troe : part == 1 ? sri : special;
            const int k1 = part == 0 ? sri : part == 1 ? c1 : troe;
            const bool spread = part < 2 && k1 - k0 <= kSpread;
            const int rank = rank_from<G>(g, part);
            #pragma unroll 1
            for (int k = k0 + (spread ? rank >> 2 : rank); k < k1; k += G) {
                const RxnEv x = load_ev(L.ev + k);
                const RxnInfo xi = load_rx(M.rx + x.r);
                SpecialK v = spread ? special_rates<4>(M, xi, s.Mtb, Tc, logT, invT, true)
                                    : special_rates(M, xi, s.Mtb, Tc, logT, invT, true);
                // non-equilibrium: the reverse Arrhenius (JacobianFunctionI.H:129-130, Jacobian.C:412-422)
                if (x.rev == 1) through_kc(x, v.Kf, v.dKfdT, v.dKfdC, v.Kr, v.dKrdT, v.dKrdC);
                if (!spread || (rank & 3) == 0) finish(x, x.r - c0, v.Kf, v.dKfdT, v.dKfdC, v.Kr, v.dKrdT, v.dKrdC);
            }
        }
        g.sync();
        const int lane = g.rank & 31, g1 = __ldg(&L.chunk[c].groupEnd);
        #pragma unroll 1
        for (int k = __ldg(&L.chunk[c].group0) + (g.rank >> 5); k < g1; k += G / 32) {
            const uint32_t e = __ldg(L.sums.elem + 32 * k + lane);
            const int m = e & 0xffff, most = __shfl_sync(0xffffffffu, m, 0), tgt = e >> 16;
            MT* o = J + (tgt >> 8) * ld + (tgt & 0xff);
            const bool valid = tgt != 0xffff;
            const double v = sum_terms(L.sums.con + __ldg(L.sums.off + k) + lane, m, most, s.q, valid ? double(*o) : 0.0);
            if (valid) *o = MT(v);
        }
        g.sync();  // the next chunk overwrites the values; the passes below read J
    }
    // third-body columns, J_ij += nu_i w_t E_tj (JF* third-body block; one
    // rounding when summing as the lane mapping does).  Up to
    // 64 threads own columns: the entries come in reaction order and a
    // reaction's products E w are formed once.  More threads than columns
    // share out the elements of the rows that have terms (one more product a
    // term, 53 species: 24,000 cycles by columns at any group size, 15,000
    // with 128 threads, 9,000 with 256).
    // (each form in a loop of its own: chosen per term, both would be issued)
    if constexpr (G <= 64) {
        #pragma unroll 1
        for (int j = g.rank; j < ns; j += G) {
            int last = -1;
            double e0 = 0, wd = 0;
            auto next_row = [&](int tb) {
                if (tb != last) {
                    e0 = __ldg(&M.eff[(size_t)tb * ns + j]);
                    wd = __dmul_rn(e0, s.tbF[tb]);
                    last = tb;
                }
            };
            if (s.rw == 1) {
                #pragma unroll 1
                for (int e = 0; e < M.nTbInc; e++) {
                    const int v = __ldg(&M.tbInc[e]), tb = (v >> 1) & 0x7fff;
                    next_row(tb);
                    const double w = s.tbF[tb];
                    MT& c = J[(v >> 16) * ld + j];
                    c = MT(fma(e0, __longlong_as_double(__double_as_longlong(w) ^ ((long long)(~v & 1) << 63)), double(c)));
                }
            } else {
                #pragma unroll 1
                for (int e = 0; e < M.nTbInc; e++) {
                    const int v = __ldg(&M.tbInc[e]);
                    next_row((v >> 1) & 0x7fff);
                    J[(v >> 16) * ld + j] += MT(__longlong_as_double(__double_as_longlong(wd) ^ ((long long)(~v & 1) << 63)));
                }
            }
        }
    } else {
        int r = g.rank / ns, j = g.rank - r * ns;
        const int dr = G / ns, dj = G - dr * ns;
        const bool once = s.rw == 1;
        while (r < M.nTbRow) {
            const int i = __ldg(M.tbRow + 2 * r), e0 = __ldg(M.tbRow + 2 * r + 1), e1 = __ldg(M.tbRow + 2 * r + 3);
            MT& o = J[i * ld + j];
            double v = double(o);
            if (once) {
                for (int e = e0; e < e1; e++) {
                    const int c = __ldg(M.tbTerm + e), tb = c >> 1;
                    v = fma(__ldg(&M.eff[(size_t)tb * ns + j]), c & 1 ? s.tbF[tb] : -s.tbF[tb], v);
                }
            } else {
                #pragma unroll 2
                for (int e = e0; e < e1; e++) {
                    const int c = __ldg(M.tbTerm + e), tb = c >> 1;
                    v += __dmul_rn(__ldg(&M.eff[(size_t)tb * ns + j]), c & 1 ? s.tbF[tb] : -s.tbF[tb]);
                }
            }
            o = MT(v);
            r += dr;
            j += dj;
            if (j >= ns) { j -= ns; r++; }
        }
    }
    // dB/dT is free now: the column factors of the conversion
    double* mj = s.dBdT;
    #pragma unroll 1
    for (int j = g.rank; j < ns; j += G) mj[j] = MW * __ldg(&M.invW[j]);
    g.sync();
    // rows: production rate and temperature column; K_i for the conversion
    double* rowK = s.dCpdT;
    #pragma unroll 1
    for (int i = g.rank; i < ns; i += G) {
        MT* row = J + i * ld;
        const double w = double(J[ns * ld + i]), tc = double(row[ns]);
        const double WiByrhoM = invRhoM * __ldg(&M.W[i]);
        const double dY = w * WiByrhoM;
        double S = 0;
        #pragma unroll 8
        for (int k = 0; k < ns; k++) S = fma(double(row[k]), s.C[k], S);
        const double tcol = WiByrhoM * (tc - S * invT) + invT * dY;
        // exact: Wi/rho (Jc_ij rho/Wj - m_j S) + m_j dY = Jc_ij (Wi/Wj) + m_j (dY - Wi/rho S)
        rowK[i] = fast ? WiByrhoM : dY - WiByrhoM * S;
        row[ns] = MT(tcol);
        f[i] = dY;
    }
    g.sync();
    // the dC/dY conversion, element by element: rows do not matter here, and
    // ns^2 elements fill the threads better than ns rows
    {
        int i = g.rank / ns, j = g.rank - i * ns;
        const int di = G / ns, dj = G - di * ns, m = ns * ns;
        #pragma unroll 1
        for (int idx = g.rank; idx < m; idx += 4 * G) {
            double w[4];
            #pragma unroll
            for (int u = 0; u < 4; u++) w[u] = !fast && idx + u * G < m ? __ldg(&M.wiw[idx + u * G]) : 0.0;
            #pragma unroll
            for (int u = 0; u < 4; u++) {
                if (idx + u * G < m) {
                    MT* e = J + i * ld + j;
                    double v;
                    if (fast) v = fma(mj[j], f[i], rowK[i] * (double(*e) * (rhoM * __ldg(&M.invW[j]))));
                    else v = fma(double(*e), w[u], mj[j] * rowK[i]);
                    *e = MT(iterate ? -v : v);
                }
                i += di;
                j += dj;
                if (j >= ns) { j -= ns; i++; }
            }
        }
    }
    double dtd = 0, dd = 0;
    if (s.rw == 1) {
        #pragma unroll 1
        for (int i = g.rank; i < ns; i += G) s.B[i] = f[i] * s.Cp[i] + double(J[i * ld + ns]) * s.Ha[i];
        serial_sums(g, ns, SumOf{s.Ha, 0, f}, SumOf{nullptr, 1.0, s.B}, s.red, dtd, dd);
    } else {
        #pragma unroll 1
        for (int i = r0; i < ns; i += s.rw) {
            const double dY = f[i], tcol = double(J[i * ld + ns]);
            dtd = fma(s.Ha[i], dY, dtd);
            dd += dY * s.Cp[i] + tcol * s.Ha[i];
        }
        gsum2(g, dtd, dd, s.red);
    }
    const double dTdt = -dtd / CpM;
    g.sync();
    // temperature row (ddTdtdYT): column owners
    #pragma unroll 1
    for (int j = g.rank; j < ns; j += G) {
        double v = 0;
        #pragma unroll 8
        for (int i = 0; i < ns; i++) {
            const double a = double(J[i * ld + j]);
            v -= (iterate ? -a : a) * s.Ha[i];
        }
        v -= s.Cp[j] * dTdt;
        const double r = v / CpM;
        J[ns * ld + j] = MT(iterate ? -r : r);
    }
    if (g.rank == 0) f[ns] = dTdt;
    if (iterate) {
        g.sync();
        #pragma unroll 1
        for (int i = g.rank; i < n; i += G) {
            const double a = i == ns ? -((-dd - dTdt * dCpMdT) / CpM) : double(J[i * ld + i]);
            J[i * ld + i] = MT(a + shift);
            if (i < ns) J[i * ld + ns] = -J[i * ld + ns];
        }
    } else if (g.rank == 0) {
        J[ns * ld + ns] = MT((-dd - dTdt * dCpMdT) / CpM);
    }
    g.sync();
}

// ------------------------------------------------------------------------
// LU with the reference's 4-row-panel pivoting (LUsolver.C:106-246 panel,
// 503-660 two- and three-row tails, 3058-3143 driver): partial pivoting
// restricted to the current panel, exact-zero pivots replaced by 2.22e-16,
// whole-row interchanges.

// t < v for v >= 0 or NaN, on the integer pipe for doubles (an FP64 compare
// costs as much as a multiply-add): the order of non-negative doubles is the
// order of their bits, a negative t sorts below them, NaN compares false.
__device__ __forceinline__ bool less_abs(double t, double v) {
    const long long a = __double_as_longlong(t), b = __double_as_longlong(v);
    return a < b && b <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool less_abs(float t, float v) { return t < v; }

// The panel's diagonal block, size x size, one element per lane: lane 4r + c
// of a warp holds a = A[r][c] (lanes 16..31 mirror 0..15).  The pivot search
// never leaves these rows, so the block is factored on its own; on return a
// holds its L and U, invD[k] the reciprocal pivots, and the result is the
// row of the panel that moved to row r.
// The loop over its columns stays rolled: unrolled per size it was no faster
// (the reciprocals' latency sets its time) and four times the code.
template<class MT>
__device__ __forceinline__ int lu_diagonal_block(MT& a, int size, double* invD, int lane) {
    const unsigned FULL = 0xffffffffu;
    const int r = (lane >> 2) & 3, c = lane & 3;
    int from = r;
    if (size == 1) {
        if (lane == 0) invD[0] = 1.0 / double(a);
        return from;
    }
    #pragma unroll 1
    for (int k = 0; k < size; k++) {
        // every lane inverts its own element while the pivot search runs; the
        // chosen row's reciprocal is then one shuffle away
        double own = double(a);
        if ((__double_as_longlong(own) << 1) == 0) own = kPivEps;
        own = double(MT(1.0 / own));
        // choose_pivot of the reference: the first column of a panel of 3 or
        // 4 rows compares all its rows, the others their own and the next
        // (the second of four also the last, LUsolver.C:169-185, where the
        // running maximum keeps the signed value of the middle row)
        int p = k;
        if (size - k > 1) {
            const MT v0 = fabs(__shfl_sync(FULL, a, 5 * k)), v1 = __shfl_sync(FULL, a, 4 * (k + 1) + k);
            const MT v2 = fabs(__shfl_sync(FULL, a, 4 * ((k + 2) & 3) + k));
            const MT v3 = fabs(__shfl_sync(FULL, a, 4 * ((k + 3) & 3) + k));
            if (k == 0 && size >= 3) {
                MT t = MT(0);
                if (less_abs(t, v0)) t = v0;
                if (less_abs(t, MT(fabs(v1)))) { p = 1; t = fabs(v1); }
                if (less_abs(t, v2)) { p = 2; t = v2; }
                if (size == 4 && less_abs(t, v3)) p = 3;
            } else if (size == 4 && k == 1) {
                MT t = v0;
                if (less_abs(t, MT(fabs(v1)))) { p = 2; t = v1; }
                if (less_abs(t, v2)) p = 3;
            } else if (less_abs(v0, MT(fabs(v1)))) {
                p = k + 1;
            }
        }
        const int src = r == k ? p : (r == p ? k : r);
        a = __shfl_sync(FULL, a, 4 * src + c);
        from = __shfl_sync(FULL, from, 4 * src + c);
        const double inv = __shfl_sync(FULL, own, 4 * p + k);
        if (lane == 0) invD[k] = inv;
        if (k + 1 < size) {
            const MT l = a * MT(inv);
            if (c == k && r > k) a = l;
            const MT lr = __shfl_sync(FULL, a, 4 * r + k), uc = __shfl_sync(FULL, a, 4 * k + c);
            const MT u = fma(-lr, uc, a);
            if (r > k && c > k) a = u;
        }
    }
    return from;
}

// One element of the trailing block: the panel's four updates.
template<class MT>
__device__ __forceinline__ MT lu_rank4(const MT* l, const MT* u, int ld, MT x) {
    return fma(-l[3], u[3 * ld], fma(-l[2], u[2 * ld], fma(-l[1], u[ld], fma(-l[0], u[0], x))));
}

// Right-looking by panels of four columns, every element's multiply-adds in
// the order of the column-by-column elimination.  Per panel, with two
// barriers: (1) threads own whole rows below the panel (their four L
// entries) and whole columns beside it (interchange, then the U entries);
// (2) the trailing block takes the panel's four updates at once, its elements
// spread over the threads row by row (m^2 / G of them each, where a fixed
// thread grid would round both dimensions up), while warp 0 updates and
// factors the next panel's diagonal block ahead of the others: that block is
// a chain of four divisions (about kAhead element updates long) which would
// otherwise keep the whole group waiting.  An FP64 instruction holds its
// scheduler for 64 cycles, so what counts is how many are issued and how
// long the group waits, not the shared-memory traffic.  Measured against the
// column-by-column form (four barriers a column, the pivot and its division
// on one thread), whole steps: 150 cells of 200 species at 256 threads
// 441 -> 288 ms, 400 of 111 species at 64 threads 82 -> 70 ms, 2,000 of 53
// species 69.3 -> 66.4 ms; 10 to 16 species unchanged (the chain of
// reciprocals sets the time there in either form).
// work: 4 ints of slot scratch that is free during the factorisation.  piv
// receives the gather permutation of the solves, (P b)[i] = b[piv[i]].
template<int G, class MT>
__device__ __noinline__ void lu_factor(const Grp<G>& g, MT* A, int n, int ld, int* piv, double* invD, int* work) {
    constexpr int W = G / 32, kAhead = 12;
    const int lane = g.rank & 31, warp = g.rank >> 5;
    const int br = (lane >> 2) & 3, bc = lane & 3;
    #pragma unroll 1
    for (int i = g.rank; i < n; i += G) piv[i] = i;
    if (warp == 0) {
        const int size = n < 4 ? n : 4;
        const bool in = br < size && bc < size;
        MT a = in ? A[br * ld + bc] : MT(0);
        const int from = lu_diagonal_block<MT>(a, size, invD, lane);
        if (in && lane < 16) A[br * ld + bc] = a;
        if (lane < 16 && bc == 0) work[br] = from;
    }
    g.sync();
    for (int k0 = 0; k0 < n; k0 += 4) {
        const int size = n - k0 < 4 ? n - k0 : 4;
        const int k1 = k0 + size, m = n - k1;
        MT* P = A + k0 * ld + k0;  // the diagonal block
        const int f0 = work[0], f1 = work[1], f2 = work[2], f3 = work[3];
        const bool moved = f0 != 0 || f1 != 1 || (size > 2 && f2 != 2);
        if (m > 0) {
            const MT r0 = MT(invD[k0]), r1 = MT(invD[k0 + 1]), r2 = MT(invD[k0 + 2]), r3 = MT(invD[k0 + 3]);
            const MT u01 = P[1], u02 = P[2], u03 = P[3], u12 = P[ld + 2], u13 = P[ld + 3], u23 = P[2 * ld + 3];
            #pragma unroll 1
            for (int i = k1 + g.rank; i < n; i += G) {
                MT* x = A + i * ld + k0;
                const MT l0 = x[0] * r0;
                MT l1 = fma(-l0, u01, x[1]), l2 = fma(-l0, u02, x[2]), l3 = fma(-l0, u03, x[3]);
                l1 *= r1;
                l2 = fma(-l1, u12, l2);
                l3 = fma(-l1, u13, l3);
                l2 *= r2;
                l3 = fma(-l2, u23, l3);
                x[0] = l0; x[1] = l1; x[2] = l2; x[3] = l3 * r3;
            }
        }
        if (m > 0 || moved) {
            // columns right of the panel, and with an interchange those left of it
            MT l10 = 0, l20 = 0, l21 = 0, l30 = 0, l31 = 0, l32 = 0;
            if (m > 0) {
                l10 = P[ld];
                l20 = P[2 * ld]; l21 = P[2 * ld + 1];
                l30 = P[3 * ld]; l31 = P[3 * ld + 1]; l32 = P[3 * ld + 2];
            }
            // the rows above took the first m threads: start with the next warp
            const int first = G == 32 ? g.rank : (g.rank + G - ((m + 31) & ~31) % G) % G;
            const int cols = moved ? m + k0 : m;
            #pragma unroll 1
            for (int t = first; t < cols; t += G) {
                MT* x = A + k0 * ld + (t < m ? k1 + t : t - m);
                MT x0 = x[f0 * ld], x1 = x[f1 * ld], x2 = size > 2 ? x[f2 * ld] : MT(0), x3 = size > 3 ? x[f3 * ld] : MT(0);
                if (t < m) {
                    x1 = fma(-l10, x0, x1);
                    x2 = fma(-l21, x1, fma(-l20, x0, x2));
                    x3 = fma(-l32, x2, fma(-l31, x1, fma(-l30, x0, x3)));
                }
                x[0] = x0;
                x[ld] = x1;
                if (size > 2) x[2 * ld] = x2;
                if (size > 3) x[3 * ld] = x3;
            }
            if (moved && g.rank == G - 1) {
                const int q0 = piv[k0 + f0], q1 = piv[k0 + f1], q2 = size > 2 ? piv[k0 + f2] : 0,
                          q3 = size > 3 ? piv[k0 + f3] : 0;
                piv[k0] = q0;
                piv[k0 + 1] = q1;
                if (size > 2) piv[k0 + 2] = q2;
                if (size > 3) piv[k0 + 3] = q3;
            }
        }
        g.sync();
        if (m == 0) break;
        const int next = m < 4 ? m : 4;
        const int iters = (m * m + 31) >> 5;
        int share = iters;  // warp 0's
        if constexpr (W > 1) {
            share = (iters - kAhead * (W - 1)) / W;
            share = share > 0 ? share : 0;
        }
        if (warp == 0) {
            const bool in = br < next && bc < next;
            MT a = MT(0);
            MT* x = A + (k1 + br) * ld + k1 + bc;
            if (in) a = lu_rank4(A + (k1 + br) * ld + k0, A + k0 * ld + k1 + bc, ld, *x);
            const int from = lu_diagonal_block<MT>(a, next, invD + k1, lane);
            if (in && lane < 16) *x = a;
            if (lane < 16 && bc == 0) work[br] = from;
        }
        {
            // two elements per step: the loads of the second overlap the
            // first's chain of multiply-adds
            const int it1 = warp == 0 ? share : iters, by = warp == 0 ? 1 : W - 1;
            int it = warp == 0 ? 0 : share + warp - 1;
            int i = (it * 32 + lane) / m, j = it * 32 + lane - i * m;
            const int di = (32 * by) / m, dj = 32 * by - di * m;
            #pragma unroll 1
            for (; it < it1; it += 2 * by) {
                int i2 = i + di, j2 = j + dj;
                if (j2 >= m) { j2 -= m; i2++; }
                const bool one = i < m && !(i < next && j < next);
                const bool two = it + by < it1 && i2 < m && !(i2 < next && j2 < next);
                MT* x = A + (k1 + i) * ld + k1 + j;
                MT* x2 = A + (k1 + i2) * ld + k1 + j2;
                MT v = 0, v2 = 0;
                if (one) v = lu_rank4(A + (k1 + i) * ld + k0, A + k0 * ld + k1 + j, ld, *x);
                if (two) v2 = lu_rank4(A + (k1 + i2) * ld + k0, A + k0 * ld + k1 + j2, ld, *x2);
                if (one) *x = v;
                if (two) *x2 = v2;
                i = i2 + di;
                j = j2 + dj;
                if (j >= m) { j -= m; i++; }
            }
        }
        g.sync();
    }
}

// Columns of one row, D at a time, and the update of one unknown by them, in order.
template<int D, class MT, class VT>
__device__ __forceinline__ VT solve_columns(const MT* row, const VT* x, int cols, int step, VT v) {
    #pragma unroll 1
    for (int c = 0; c < cols; c += D) {
        MT a[D];
        VT y[D];
        #pragma unroll
        for (int q = 0; q < D; q++) {
            const int k = (c + q < cols ? c + q : c) * step;
            a[q] = row[k];
            y[q] = x[k];
        }
        #pragma unroll
        for (int q = 0; q < D; q++)
            if (c + q < cols) v = fma(-VT(a[q]), y[q], v);
    }
    return v;
}

// Forward/back substitution with the factors of lu_factor after the row
// interchanges (LUsolver.C:3145-3171, 4113-4152), every unknown's
// multiply-adds in the order of the column sweeps.  b is a slot vector;
// arithmetic in VT.
//
// By blocks of 32 unknowns, one warp's lanes: within a block the solved
// unknown goes from its lane to the others by shuffle and the matrix elements
// are loaded ahead, so that a column costs the chain of its FP64 operations
// (95 cycles forward, 160 backward with the multiplication by the reciprocal
// pivot) instead of a round trip through shared memory.  Blocks belong to the
// warps in turn; the owner of the next block brings it up to date first and
// solves it while the other warps update the blocks behind it, one barrier a
// block.  Cycles per solve, one cell per SM, against one warp sweeping whole
// columns: 53 species, 64 threads 36,500 -> 26,400; 111 species, 256 threads
// 99,000 -> 58,000; 200 species (global workspace), 256 threads 796,000 ->
// 188,000.  Six 53-species cells per SM: 40,800 -> 30,500.
template<int D, int G, class MT, class VT>
__device__ __noinline__ void lu_solve_ahead(const Grp<G>& g, const MT* A, int n, int ld, const int* perm,
                                            const double* invD, VT* b) {
    constexpr int W = G / 32, U = (256 + G - 1) / G;
    const unsigned FULL = 0xffffffffu;
    const int lane = g.rank & 31, warp = g.rank >> 5, nb = (n + 31) >> 5;
    g.sync();
    {
        VT t[U];
        #pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = g.rank + G * u;
            t[u] = i < n ? b[perm[i]] : VT(0);
        }
        g.sync();
        #pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = g.rank + G * u;
            if (i < n) b[i] = t[u];
        }
    }
    g.sync();
    // forward, unit lower triangle
    #pragma unroll 1
    for (int kb = 0; kb < nb; kb++) {
        const VT* x = b + 32 * (kb - 1);  // the block solved last
        if (kb % W == warp) {
            const int i = 32 * kb + lane, cols = n - 32 * kb < 32 ? n - 32 * kb : 32;
            const MT* row = A + (i < n ? i : n - 1) * ld;
            VT v = b[i < n ? i : n - 1];
            if (kb > 0) v = solve_columns<D, MT, VT>(row + 32 * (kb - 1), x, 32, 1, v);
            #pragma unroll 1
            for (int c = 0; c < cols; c += D) {
                MT a[D];
                #pragma unroll
                for (int q = 0; q < D; q++) a[q] = row[32 * kb + (c + q < cols ? c + q : c)];
                #pragma unroll
                for (int q = 0; q < D; q++) {
                    if (c + q < cols - 1) {
                        const VT xj = __shfl_sync(FULL, v, c + q);
                        const VT w = fma(-VT(a[q]), xj, v);
                        if (lane > c + q) v = w;
                    }
                }
            }
            if (i < n) b[i] = v;
        }
        if (kb > 0) {
            int rb = kb + 1 + (warp - (kb + 1) % W + W) % W;  // this warp's next block after kb
            #pragma unroll 1
            for (; rb < nb; rb += W) {
                const int i = 32 * rb + lane;
                if (i < n) b[i] = solve_columns<D, MT, VT>(A + i * ld + 32 * (kb - 1), x, 32, 1, b[i]);
            }
        }
        if (kb + 1 < nb) g.sync();
    }
    // backward, upper triangle and reciprocal pivots
    #pragma unroll 1
    for (int kb = nb - 1; kb >= 0; kb--) {
        const int last = kb + 1 < nb ? (n - 32 * (kb + 1) < 32 ? n - 1 : 32 * (kb + 1) + 31) : 0;
        const int had = last - 32 * (kb + 1) + 1;  // unknowns of the block solved last
        if (kb % W == warp) {
            const int i = 32 * kb + lane, cols = n - 32 * kb < 32 ? n - 32 * kb : 32;
            const MT* row = A + (i < n ? i : n - 1) * ld;
            VT v = b[i < n ? i : n - 1];
            if (kb + 1 < nb) v = solve_columns<D, MT, VT>(row + last, b + last, had, -1, v);
            const VT inv = VT(invD[i < n ? i : n - 1]);
            #pragma unroll 1
            for (int c = cols - 1; c >= 0; c -= D) {
                MT a[D];
                #pragma unroll
                for (int q = 0; q < D; q++) a[q] = row[32 * kb + (c - q >= 0 ? c - q : c)];
                #pragma unroll
                for (int q = 0; q < D; q++) {
                    if (c - q >= 0) {
                        const VT xj = __shfl_sync(FULL, v * inv, c - q);
                        const VT w = fma(-VT(a[q]), xj, v);
                        v = lane < c - q ? w : (lane == c - q ? xj : v);
                    }
                }
            }
            if (i < n) b[i] = v;
        }
        if (kb + 1 < nb) {
            int rb = warp;
            #pragma unroll 1
            for (; rb < kb; rb += W) {
                const int i = 32 * rb + lane;
                b[i] = solve_columns<D, MT, VT>(A + i * ld + last, b + last, had, -1, b[i]);
            }
        }
        if (kb > 0) g.sync();
    }
    g.sync();
}

// Loads of eight columns ahead hide the latency of a slot in L2 (201 unknowns,
// 256 threads: 144,000 cycles, with four 178,000); in shared memory four give
// the same time (54 unknowns: 25,500 and 25,900 cycles) in half the code, which
// counts where small groups fill an SM.
template<int G, class MT, class VT>
__device__ __forceinline__ void lu_solve(const Grp<G>& g, const MT* A, int n, int ld, const int* perm,
                                         const double* invD, VT* b) {
    if constexpr (G < 256) {
        if (__isShared(A)) return lu_solve_ahead<4, G, MT, VT>(g, A, n, ld, perm, invD, b);
    }
    lu_solve_ahead<8, G, MT, VT>(g, A, n, ld, perm, invD, b);
}

}  // namespace fcs
