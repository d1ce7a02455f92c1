// cueva_common.cuh -- shared definitions of the B200 CUEVA kernels.
//
// Device data layout (HBM): structure of arrays, one slab per field group,
// interior points only.  Point (i, j), 0 <= i <= imax, 0 <= j <= jmax, of
// field f lives at base + f * fstride + j * pitch + i, with pitch a multiple
// of 32 doubles (256 B rows) so every warp-wide row access is one aligned
// 256 B segment.  Ghost cells of the Fortran arrays are never stored: loads
// outside the interior go through the per-axis index map of the reference's
// boundary routines (copy = clamp to [0, N]; periodic = node duplicate,
// -k -> N-k and N+k -> k; 04_boundary.f95:1390-1533, 2867-3033).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace cueva {

// ---- field groups --------------------------------------------------------
// carried primitive state, order of the C-ABI prims (include/cueva.h)
enum Prim { P_RHO = 0, P_P, P_VX, P_VY, P_VZ, P_PSI, P_PHI, P_EX, P_EY, P_EZ, P_BX, P_BY, P_BZ, P_Q, NPRIM };
// conserved D, tau, S and the Lorentz factor at time n (startconvar)
enum Aux { A_D = 0, A_TAU, A_SX, A_SY, A_SZ, A_W, NAUX };
// RK stage state: the 14 conserved of stage l (E already implicit) + J
enum Stage { Q_PSI = 0, Q_PHI, Q_EX, Q_EY, Q_EZ, Q_BX, Q_BY, Q_BZ, Q_Q, Q_D, Q_TAU, Q_SX, Q_SY, Q_SZ,
             Q_JX, Q_JY, Q_JZ, NSTAGE };
constexpr int NCONS = 14;   // first 14 stage fields are the conserved set
// stage right-hand side: F (14, same order as the conserved set) + E sources
enum Rhs { K_SEX = 14, K_SEY, K_SEZ, NRHS };

// ---- status bits (host maps them to C-ABI error codes) -------------------
enum StatusBits : uint32_t {
  ST_C2P_FAIL = 1u,        // Cardano "stop" branches, 12_varprimitive.f95:382-428,485
  ST_SUPERLUMINAL = 2u,    // 12_varprimitive.f95:678,691 ; 12_varprimitive_nr.f95:217
  ST_HLLC_NOCONV = 4u,     // funciones.f95:240-245
  ST_HLLC_VSTAR = 8u,      // 16_hllc_flow_mpx.f95:4294,4605
  ST_NONFINITE = 16u,      // con2prim returned NaN / Inf
  ST_HLLE_SPEED = 32u,     // 16_hlle_flow_mpx.f95:2796-2803, 2974-2981
  ST_TC_TIMEOUT = 64u,     // a bounded tensor-core wait ran out (no reference counterpart)
  ST_TC_TEARDOWN = 128u,   // after such a time-out the teardown's bounded wait for the MMAs still in
                           // flight ran out too: TMEM was released while an MMA may still write it, so
                           // the context is suspect and should not be reused
  ST_COPY_TIMEOUT = 256u,  // a bounded wait for the bulk copies of the stage kernel's stencil rows ran
                           // out (no reference counterpart); the CTA stopped
};

// ---- per-instance descriptor (one grid of the ensemble) -------------------
struct InstDesc {
  // device buffers
  double* prim[2];     // double-buffered NPRIM slabs
  double* aux[2];      // double-buffered NAUX slabs
  double* stage[2];    // double-buffered NSTAGE slabs
  double* intsum;      // NCONS slab (needed when the tableau has >= 3 stages)
  double* finsum;      // NCONS slab
  double* kbuf;        // nk * NRHS slabs of stored stage right-hand sides
  double* rhs_out;     // NRHS slab written in the store-rhs mode
  uint32_t* status;    // status word
  unsigned long long* counters;  // [3] fix-up counters (rho, p, v)
  // learned con2prim seed network (null unless c2p method 2)
  const void* mlp;
  // geometry
  int imax, jmax;      // interior points 0..imax, 0..jmax
  int pitch;           // doubles per row
  long long fstride;   // doubles per field slab
  int bc_x, bc_y;      // 0 copy, 1 periodic
  // scalars
  double delx, dely, dt, sigma, gamma, kappa_psi, kappa_phi;
  // 1/delx, 1/dely when the spacing is a power of two (then v * inv == v / del
  // exactly and the divisions of the flux divergence become multiplications);
  // 0 otherwise
  double inv_delx_pow2, inv_dely_pow2;
  double recip_delx, recip_dely;   // RN(1/delx), RN(1/dely) (divide_spacing)
  double eps1_c2p;     // value of the Fortran module variable eps1 when con2prim runs
  int c2p;             // 1 Cardano, 0 NR, 2 learned seed + Newton (Cardano fallback)
  int primitive_rec;   // 1: the step starts with the primitive reconstruction (k_recons_begin),
                       // so the last stage does not prepare the next step's stage 1
  int c2p_tc;          // c2p 2 with a network: 1 = con2prim in k_c2p_step on the tcgen05 tensor
                       // cores after the last stage, 0 = inside the last stage (warp mma.sync)
  // interface flux scratch: Fx(i+1/2, j) at fx[(j) * fpitch + (i + 1)],
  // Fy(i, j+1/2) at fy[(j + 1) * fpitch + i], NFACE fields each
  double* fx;
  double* fy;
  int fpitch;
  long long ffs;       // doubles per flux field
  // work decomposition: tiles of each launch kind (x faces + update, y faces,
  // learned con2prim, fused stage)
  int block_begin[4];
  int block_count[4];
  int seg_rows;        // fused stage tiles: grid rows per tile (bands of the tile height, less one row)
};

// ---- tableau data of one stage launch (by value, kernel parameter space) -----
struct StageArgs {
  int l;               // 1-based RK stage being swept
  int s;               // number of stages
  int cur;             // which prim/aux buffer holds time n
  int qin;             // which stage buffer holds stage l
  double wb, wbt;      // wb(l), wbt(l)
  double ab_next[8];   // Ab(l+1, 1..l)
  double abt_next[8];  // Abt(l+1, 1..l)
  double abt_diag_next;// Abt(l+1, l+1)
  double abt_diag_first;// Abt(1,1) (next step's stage 1)
  int kslot[8];        // slot of stored K_m in kbuf, -1 if not stored
  int store_k_slot;    // slot to store K_l, -1 if not needed
  int store_k_src;     // K_l is only read through its E sources (every later row has Ab = 0 in
                       // column l): store the 3 sources, not the 14 fluxes
  int fin_load;        // the final sums of earlier stages are not all zero (some wb, wbt of m < l
                       // is non-zero): load them; else they start from zero
  int fin_store;       // the final sums after this stage are not identically zero: store them
  int need_intsum_load;  // stage l >= 2 and s >= 3: intsum_l is stored
  int need_intsum_store; // l + 1 < s
  int mode;            // 0 fused (next stage / final), 1 store rhs only, 2 also the x-face fluxes (I.fx)
  double* diag_cons;   // last stage: D and tau of varfin stored here (2 slabs) when non-null
};

// ---- small math helpers (Fortran semantics) ------------------------------
template <typename T> __device__ __forceinline__ T pw2(T x) { return x * x; }
template <typename T> __device__ __forceinline__ T pw3(T x) { return (x * x) * x; }
template <typename T> __device__ __forceinline__ T pw4(T x) { T t = x * x; return t * t; }
template <typename T> __device__ __forceinline__ T fmin2(T a, T b) { return (b < a) ? b : a; }
template <typename T> __device__ __forceinline__ T fmax2(T a, T b) { return (b > a) ? b : a; }
template <typename T> __device__ __forceinline__ T fsgn1(T b) { return copysign(T(1), b); }

// ---- several divisions by one divisor ---------------------------------------
// divide_all replaces each a[k] by the correctly rounded a[k] / b, given the
// correctly rounded reciprocal z of b: q = RN(a z), r = a - q b (exact in an
// FMA), RN(q + r z) -- three operations per quotient where a division takes a
// dozen and its own reciprocal (Brisebarre, Muller & Raina, "Accelerating
// correctly rounded floating-point division when the divisor is known in
// advance", IEEE Trans. Computers 53, 2004).  The sign is taken from a, so
// that signed zeros come out as the division gives them (b > 0, or b's
// sign).  Exact while nothing under- or overflows on the way: the exponents
// of b and of every nonzero a are tested (magnitude_key: a subnormal whose
// high word is zero is no zero), and values out of range take the division
// itself, in a rolled loop (they are rare, and the code stays small).
// Used for the 28 flux differences of a point where a spacing is no power of
// two, and the 14 star-state quotients of an HLLC face.  Steps on a B200,
// divisions one by one -> shared: 500 x 1000 HLL + MC 433 -> 361 us, 700 x
// 1500 HLLC + MP9 2.91 -> 2.41 ms, 611 x 1003 HLL + MP7 1214 -> 1001 us, 2048 x
// 4096 HLLC + MP5 (power-of-two spacings) 16.24 -> 15.43 ms.  Telling subnormals
// from zeros by their low words costs 0.5 to 1 % of a step (13.92 -> 13.99 ms
// at 2048 x 4096, 359 -> 362 us at 500 x 1000 HLL + MC).
__device__ __forceinline__ double recip_rn(double b) { return __drcp_rn(b); }
__device__ __forceinline__ float recip_rn(float b) { return __frcp_rn(b); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// sign and exponent bits of a value, and the range of |a| and |b| in them
__device__ __forceinline__ uint32_t high_word(double x) { return (uint32_t)__double2hiint(x); }
__device__ __forceinline__ uint32_t high_word(float x) { return __float_as_uint(x); }
// |x| by its leading bits, zero for zeros alone
__device__ __forceinline__ uint32_t magnitude_key(double x) {
  return (high_word(x) & 0x7fffffffu) | min((uint32_t)__double2loint(x), 1u);
}
__device__ __forceinline__ uint32_t magnitude_key(float x) { return high_word(x) & 0x7fffffffu; }
template <typename T> struct DivRange;
template <> struct DivRange<double> {   // a in 2^-800 .. 2^800, b in 2^-100 .. 2^100
  static constexpr uint32_t a_lo = (1023u - 800u) << 20, a_hi = (1023u + 800u) << 20;
  static constexpr uint32_t b_lo = (1023u - 100u) << 20, b_hi = (1023u + 100u) << 20;
};
template <> struct DivRange<float> {    // a in 2^-80 .. 2^60, b in 2^-40 .. 2^40
  static constexpr uint32_t a_lo = (127u - 80u) << 23, a_hi = (127u + 60u) << 23;
  static constexpr uint32_t b_lo = (127u - 40u) << 23, b_hi = (127u + 40u) << 23;
};
__device__ __forceinline__ double with_sign(double m, uint32_t s) {
  return __hiloint2double((int)((high_word(m) & 0x7fffffffu) | (s & 0x80000000u)), __double2loint(m));
}
__device__ __forceinline__ float with_sign(float m, uint32_t s) {
  return __uint_as_float((__float_as_uint(m) & 0x7fffffffu) | (s & 0x80000000u));
}
template <int N, typename T>
__device__ __forceinline__ void divide_all(T (&a)[N], T b, T z) {
  const uint32_t hb = high_word(b);
  uint32_t lo = 0xffffffffu, hi = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const uint32_t h = magnitude_key(a[k]);
    lo = min(lo, h - 1u);   // a zero passes
    hi = max(hi, h);
  }
  if (lo >= DivRange<T>::a_lo - 1u && hi <= DivRange<T>::a_hi &&
      (hb & 0x7fffffffu) - DivRange<T>::b_lo <= DivRange<T>::b_hi - DivRange<T>::b_lo) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const T q = a[k] * z;
      a[k] = with_sign(fma_rn(fma_rn(-b, q, a[k]), z, q), high_word(a[k]) ^ hb);
    }
  } else {
    T t[N];
#pragma unroll
    for (int k = 0; k < N; ++k) t[k] = a[k];
#pragma unroll 1
    for (int k = 0; k < N; ++k) t[k] = t[k] / b;
#pragma unroll
    for (int k = 0; k < N; ++k) a[k] = t[k];
  }
}
// differences of a flux divergence over a grid spacing: inv_pow2 as in
// InstDesc, recip the spacing's reciprocal
template <int N>
__device__ __forceinline__ void divide_spacing(double (&d)[N], double spacing, double inv_pow2, double recip) {
  if (inv_pow2 != 0.0) {
#pragma unroll
    for (int k = 0; k < N; ++k) d[k] = d[k] * inv_pow2;
  } else {
    divide_all(d, spacing, recip);
  }
}

// ghost index maps of the reference's boundary routines
__device__ __forceinline__ int map_idx(int i, int n, int periodic) {
  if (i < 0) return periodic ? i + n : 0;
  if (i > n) return periodic ? i - n : n;
  return i;
}

// launch geometry: 32 x ROWS threads per CTA for the face tiles (x tiles
// update 31 points per row; ROWS is 8 or 4), 256 threads for the pointwise
// kernels
constexpr int FACE_ROWS = 8;   // default tile height
constexpr int WIDE_ROWS = 12;  // most warps of a tile of the fused stage kernel's wide form
constexpr int NFACE = 14;   // interface fluxes per face (the Riemann roles)
constexpr int POINT_THREADS = 256;
enum LaunchKind { LK_XUPD = 0, LK_YFACE = 1, LK_C2P = 2, LK_STAGE = 3 };

// launch shape of one RK stage: tile height, CTAs per launch kind and the
// tiles they loop over (grid == ntiles: one tile per CTA; smaller: persistent).
// fused: the stage runs as one k_stage launch (grid[LK_STAGE] CTAs over
// ntiles[LK_STAGE] tiles) instead of k_yface + k_xupd.
struct StageShape {
  int rows = FACE_ROWS;
  int grid[4] = {0, 0, 0, 0};
  int ntiles[4] = {0, 0, 0, 0};
  bool fused = false;
  // not 0: one k_stage per stage in its wide form, with this many warps per tile
  // (ntiles[LK_STAGE] tiles of one row less): see stage_wide_rows
  int wide_rows = 0;
};

// tiles of one instance for a tile height (x tiles: 31 points by rows)
inline int xupd_tiles(int imax, int jmax, int rows) { return ((imax + 1 + 30) / 31) * ((jmax + 1 + rows - 1) / rows); }
inline int yface_tiles(int imax, int jmax, int rows) { return ((imax + 1 + 31) / 32) * ((jmax + 2 + rows - 1) / rows); }
// fused stage tiles: strips of 31 points by segments of seg_rows grid rows
inline int stage_tiles(int imax, int jmax, int seg_rows) {
  return ((imax + 1 + 30) / 31) * ((jmax + 1 + seg_rows - 1) / seg_rows);
}

// The mixed-precision flux routines keep the fluxes of the field roles psi,
// phi, Bn, Bt1, Bt2, En, Et1, Et2 (roles 0..7) in FP64: they carry the
// uniform background field (B ~ 0.1 in the KH runs), whose FP32 rounding
// (~4e-9) is not small against E itself, and the final IMEX combination
// passes that error into E(n+1) undamped.  All routines but HLLE-MC
// (flux_solver 3, whose field star states use the sound-speed bounds).
__host__ __device__ constexpr bool mixed_em_f64(int solver) { return solver >= 1 && solver <= 7 && solver != 3; }
// The mixed-precision MP routines HLL, HLLE and HLLC (flux_solver 5..7) also
// form the normal momentum flux in FP64: its pressure part, ~1 in the KH
// layer, is added to the FP32 rest there (see the split pressure of the
// stage kernels).
__host__ __device__ constexpr bool mixed_split_p(int solver) { return solver >= 5 && solver <= 7; }
constexpr int ROLE_SN = 11;   // the normal momentum flux (R_SN of the Riemann roles)

// Place of role r in the y-flux scratch (NFACE slabs of ffs doubles): f64
// tells the element type and off the slab's first element in units of that
// type.  FP64 kernels: double slab r.  Mixed kernels: FP32 slab r; with
// mixed_em_f64, double slabs 0..7 for roles 0..7, then FP32 slabs for roles
// 8..13 from byte offset 64 * ffs on; with mixed_split_p also, the normal
// momentum flux in double slab 8 and the other five FP32 slabs from byte
// offset 72 * ffs on.
struct FluxSlot {
  bool f64;
  long long off;
};
__host__ __device__ inline FluxSlot flux_slot(bool mixed, int solver, int r, long long ffs) {
  if (!mixed) return {true, r * ffs};
  if (!mixed_em_f64(solver)) return {false, r * ffs};
  if (r <= 7) return {true, r * ffs};
  if (mixed_split_p(solver)) {
    if (r == ROLE_SN) return {true, 8 * ffs};
    return {false, (18 + (r < ROLE_SN ? r - 8 : r - 9)) * ffs};
  }
  return {false, (16 + (r - 8)) * ffs};
}

}  // namespace cueva
