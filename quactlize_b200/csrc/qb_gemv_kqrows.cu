// Raw k-quant blocks (Q2_K .. Q6_K), up to eight activation rows per pass over the weights, dense and ragged MoE, rows of
// any byte alignment the format allows.
//
//   out[t, r] = sum_b ( d_rb * sum_g sc_rbg * sum_j q_rbgj x[t, ..]  -  dmin_rb * sum_g mn_rbg * sum_j x[t, ..] )
//
// Same contract as vecdot_rows_kernel of the reference for M > 1 and for its grouped launches
// (quactlize/include/gguf_vecdot.hpp:604-760, launch policy :564-602).
//
// Arithmetic.  sub-scale x code is an integer of at most 11 bits in every format (63*31 for Q5_K; Q6_K is two such
// products, sc*lo4 and 16*sc*(hi2 - 2)), so it is EXACT in fp16: the masked word (w & 0x000F000F, a half2 of fp16
// subnormals q * 2^-24) times the sub-scale is an A fragment of mma.sync.m16n8k16 and all 256 codes of a superblock go
// into one fp32 accumulator tile, scaled by d once.  The B fragments are the fp16 activations as they are.  Which code
// feeds which k index is free as long as A and B agree, so a lane reads its own 16-byte chunk of a weight row and needs
// the sub-scales of four groups only, with no exchange between lanes.  Sub-mins: two (Q2_K: three) bf16 MMAs against the
// per-group sums of x, the fp32 sums whole as three bf16 parts of 8 bits; the sums come from 16 MMAs with an indicator matrix.
//
// Rounding.  An MMA cuts its fp32 sum off where a fused multiply-add rounds, and it lines its products up by their exponent
// fields, so an fp16 subnormal costs the sum as many bits as it has leading zeros.  The sub-scales therefore carry a power of two
// (kr_up) that lifts the products out of the subnormals, a chain of MMAs is at most four long before its sum goes to a rounded
// add, and a tile's K slices are added even and odd apart.  Relative error against 64 bits, N(0,1) activations, K 1280 to
// 14336, against 22-bit group sums, chains of eight (Q6_K sixteen) and no lift: Q2_K 2.2e-7 -> 0.8e-7, Q3_K 1.2e-7 -> 0.8e-7,
// Q4_K 1.8e-7 -> 1.2e-7, Q5_K 2.0e-7 -> 1.3e-7; 4096 -> 14336, us: Q2_K 8 rows 14.9 -> 13.1, Q3_K 4 rows 15.9 -> 16.2, Q4_K 8 rows
// 13.2 -> 13.0, Q5_K 4 rows 16.3 -> 16.2.  Q6_K, two products a code, has its chains cut only where a rounded kernel
// was before it: rows off a 16-byte boundary 2.3e-7 -> 1.0e-7 (4096 x 2304, three rows 8.0 -> 9.0 us; the plain kernel 0.8e-7 and 38 us);
// its other rows took the one-row kernel's 8e-4 before and keep 2.3e-7.
//
// Structure.  One CTA per SM: 16 computing warps, a copy warp, a reducing warp.  K is covered in passes of P superblocks,
// and for deep rows cut over the CTAs of a cluster; warp (slot, b) owns superblock b of the pass and keeps its B fragments
// in registers over all tiles; a ring stage is RS tiles of 16 rows x P superblocks, one cp.async.bulk per row (rows off a
// 16-byte boundary are copied from the boundary below, and nothing outside the tensor is read).  The activations of a pass arrive through shared memory the same
// way, a pass ahead (the very first ones by plain loads).  The K slices of a tile are added in warp order, then in CTA order, by the reducing warp (results do
// not depend on timing) while the others work on the next tile.  The tiles of all (expert, eight-row group) pairs form one
// list that is cut evenly over the clusters: empty experts cost nothing and a launch is one wave whatever the router does.
//
// Rows of 84-, 110- and 210-byte blocks are read in 4-byte words, the word order rotated by the lane's quarter: rows lie
// 16 bytes off a 128-byte pitch, so the 32 lanes of a load fall on 32 banks.  Every wait is bounded.
//
// Measured, 4096 -> 14336, eight rows, us: Q4_K 15.5 -> 13.0 (33 MB, 2.6 TB/s), Q2_K 41 -> 13.1, Q3_K 64 -> 16.4, Q5_K 58 -> 16.6,
// Q6_K 66 -> 19.7.  What bounds it is the latency of a tile round, about 1.1 us for Q4_K against 0.83 us of stream: about 260
// instructions a warp, half of them on the half-rate integer pipe, with four to five warps per scheduler.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>

#include "qb_device.cuh"
#include "qb_internal.hpp"
#include "qb_kqrows_units.hpp"
#include "qb_kquant.cuh"
#include "qb_runtime.hpp"

namespace qb {
namespace {

constexpr int kKrWarps = 16;                       // computing warps
constexpr int kKrThreads = (kKrWarps + 2) * 32;
constexpr int kKrTile = 16;
constexpr int kKrMaxStages = 8;
constexpr int kKrMaxExperts = 4096;                // their offsets and group counts: 32 KB of shared memory at most
constexpr int kKrAccTiles = 16;                    // tiles whose sums the reducing warp carries over K passes and CTAs
// The first activations of a CTA by plain loads of the computing warps: 0.3 us earlier than through shared memory at one to
// four rows (Q4_K 2400 x 4096, 2 rows: 6.05 against 6.43 us), later at eight (14336 x 4096: 13.3 against 12.9 us).
constexpr int kKrDirectRows = 4;
constexpr size_t kKrSmem = 227 * 1024;

struct KrArgs {
  uint8_t const* blocks;
  __half const* x;
  float* out;
  int const* offsets;                              // cumulative [experts+1] (grouped) or nullptr
  int n, bpr, experts, m_rows;
  int passes, P, RS, C;                            // K passes, superblocks per pass, tiles per ring stage, CTAs that share K
  int pitch, xpitch, xrows, stages, xbufs, tiles, round;   // round: tiles of a segment at most
  unsigned int* status;
};

__device__ __forceinline__ uint32_t kr_lds32(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t kr_lds16(uint32_t a) { uint16_t v; asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint2 kr_lds64(uint32_t a) { uint2 v; asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); return v; }
__device__ __forceinline__ uint4 kr_lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void kr_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// D = A * B: the first of a chain
__device__ __forceinline__ void kr_mma0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void kr_mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void kr_mma_bf16_k8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(b0));
}
// power of two on the scaled codes: the largest whose constant in kr_scale is an fp16 number, with 16 * sc in Q6_K's range
template <int QT> constexpr float kr_up() { return QT == 14 ? 16.f : 32.f; }
__device__ __forceinline__ __half2 kr_mask(uint32_t w, uint32_t m) { return u32_as_h2(w & m); }
// byte `idx` of w, as half2 (b + add) * mul in both lanes; exact for the values used here
__device__ __forceinline__ __half2 kr_scale(uint32_t w, uint32_t idx, float mul, float add) {
  return __hfma2(u32_as_h2(__byte_perm(w, 0x64646464u, 0x4040u + 0x0101u * idx)), __float2half2_rn(mul), __float2half2_rn((add - 1024.f) * mul));
}
// bytes 2p, 2p+1 of w, below 128, as a bf16 pair: 128 + b has b in its mantissa
__device__ __forceinline__ uint32_t kr_min_pair(uint32_t w, uint32_t p) {
  uint32_t v = __byte_perm(w, 0x43434343u, 0x4140u + 0x0202u * p);
  __nv_bfloat162 const m = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&v), __float2bfloat162_rn(128.f));
  return *reinterpret_cast<uint32_t const*>(&m);
}

// One weight row's share of a lane: the words, one sub-scale multiplier per field, the header.  load() reads it; frag(j, wi)
// are the A registers of (field j, word wi): elements (0, 2) and (1, 3) of the word, times the field's sub-scale.
template <int QT> struct KrRow;

template <> struct KrRow<12> {                                      // Q4_K
  uint32_t q[2][4];
  __half2 s[4];
  float d, dmin;
  uint32_t mn[1];                                                   // sub-mins of groups 2t, 2t+1
  __device__ __forceinline__ void load(uint32_t sb, int t) {
    uint4 const h = kr_lds128(sb);
    codes(sb + 16 + 16 * t);
    header(h, t);
  }
  __device__ __forceinline__ void codes(uint32_t a) {
    uint4 const q0 = kr_lds128(a), q1 = kr_lds128(a + 64);
    q[0][0] = q0.x; q[0][1] = q0.y; q[0][2] = q0.z; q[0][3] = q0.w;
    q[1][0] = q1.x; q[1][1] = q1.y; q[1][2] = q1.z; q[1][3] = q1.w;
  }
  __device__ __forceinline__ void header(uint4 h, int t) {
    float2 const dd = __half22float2(u32_as_h2(h.x));
    d = dd.x; dmin = dd.y;
    uint32_t const sc_lo = h.y & 0x3F3F3F3Fu, sc_hi = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
    uint32_t const mn_lo = h.z & 0x3F3F3F3Fu, mn_hi = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
    uint32_t const i0 = uint32_t(t & 2);                            // the chunk's even group within its word
    constexpr float up = kr_up<12>();
    s[0] = kr_scale(sc_lo, i0, up, 0.f); s[1] = kr_scale(sc_lo, i0 + 1, up * 0.0625f, 0.f);
    s[2] = kr_scale(sc_hi, i0, up, 0.f); s[3] = kr_scale(sc_hi, i0 + 1, up * 0.0625f, 0.f);
    mn[0] = kr_min_pair((t & 2) ? mn_hi : mn_lo, uint32_t(t & 1));
  }
  __device__ __forceinline__ void frag(int j, int wi, uint32_t (&a)[2]) const {
    uint32_t const w = q[j >> 1][wi], m = (j & 1) ? 0x00F000F0u : 0x000F000Fu;
    a[0] = h2_as_u32(__hmul2(kr_mask(w, m), s[j]));
    a[1] = h2_as_u32(__hmul2(kr_mask(w >> 8, m), s[j]));
  }
};

template <> struct KrRow<13> : KrRow<12> {                          // Q5_K: the fifth bit on top
  uint32_t hb[4];
  __half2 sh[4];
  __device__ __forceinline__ void load(uint32_t sb, int t) {
    uint4 const h = kr_lds128(sb), b = kr_lds128(sb + 16 + 16 * (t & 1));
    codes(sb + 48 + 16 * t);
    int const pre = t & 2;                                          // bits of groups 0,1,4,5 relative to the lane's first group
    hb[0] = b.x >> pre; hb[1] = b.y >> pre; hb[2] = b.z >> pre; hb[3] = b.w >> pre;
    header(h, t);
    sh[0] = __hmul2(s[0], __float2half2_rn(16.f)); sh[1] = __hmul2(s[1], __float2half2_rn(128.f));   // sc*16 / 2^bit
    sh[2] = s[2];                                  sh[3] = __hmul2(s[3], __float2half2_rn(8.f));
  }
  __device__ __forceinline__ void frag(int j, int wi, uint32_t (&a)[2]) const {
    uint32_t const w = q[j >> 1][wi], m = (j & 1) ? 0x00F000F0u : 0x000F000Fu;
    uint32_t const hm = 0x00010001u << (4 * (j >> 1) + (j & 1));
    a[0] = h2_as_u32(__hfma2(kr_mask(hb[wi], hm), sh[j], __hmul2(kr_mask(w, m), s[j])));
    a[1] = h2_as_u32(__hfma2(kr_mask(hb[wi] >> 8, hm), sh[j], __hmul2(kr_mask(w >> 8, m), s[j])));
  }
};

template <> struct KrRow<10> {                                      // Q2_K (4-byte aligned blocks)
  uint32_t q[4];
  __half2 s[4];
  float d, dmin;
  uint32_t mn[2];                                                   // sub-mins of groups 2t, 2t+1 and 2t+8, 2t+9
  __device__ __forceinline__ void load(uint32_t sb, int t) {
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = kr_lds32(sb + 16 + 16 * t + 4 * ((i + t) & 3));
    uint32_t const w0 = kr_lds32(sb), w1 = kr_lds32(sb + 4), w2 = kr_lds32(sb + 8), w3 = kr_lds32(sb + 12);
    float2 const dd = __half22float2(u32_as_h2(kr_lds32(sb + 80)));
    d = dd.x; dmin = dd.y;
    uint32_t const sa = ((t & 2) ? w2 : w0) & 0x0F0F0F0Fu, sc = ((t & 2) ? w3 : w1) & 0x0F0F0F0Fu, p = uint32_t(t & 1);
    constexpr float up = kr_up<10>();
    s[0] = kr_scale(sa, p, up, 0.f);              s[1] = kr_scale(sa, p + 2, up * 0.25f, 0.f);
    s[2] = kr_scale(sc, p, up * 0.0625f, 0.f);    s[3] = kr_scale(sc, p + 2, up * 0.015625f, 0.f);
    mn[0] = kr_min_pair((((t & 2) ? w1 : w0) >> 4) & 0x0F0F0F0Fu, p);
    mn[1] = kr_min_pair((((t & 2) ? w3 : w2) >> 4) & 0x0F0F0F0Fu, p);
  }
  __device__ __forceinline__ void frag(int j, int wi, uint32_t (&a)[2]) const {
    uint32_t const m = 0x00030003u << (2 * j);
    a[0] = h2_as_u32(__hmul2(kr_mask(q[wi], m), s[j]));
    a[1] = h2_as_u32(__hmul2(kr_mask(q[wi] >> 8, m), s[j]));
  }
};

// four words at byte address `a` (2-byte aligned), in the rotated order
__device__ __forceinline__ void kr_run(uint32_t a, int t, uint32_t (&w)[4]) {
  uint32_t const b = a & ~3u, sh = (a & 2u) * 8u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t const p = b + 4 * ((i + t) & 3);
    w[i] = __funnelshift_r(kr_lds32(p), kr_lds32(p + 4), sh);
  }
}

template <> struct KrRow<11> {                                      // Q3_K (2-byte aligned blocks)
  uint32_t q[4], nb[4];                                             // 2-bit fields; inverted high bits of the lane's half
  __half2 s[4], sn[4];
  float d;
  __device__ __forceinline__ void load(uint32_t sb, int t) {
    kr_run(sb + 32 + 16 * t, t, q);
    kr_run(sb + 16 * (t & 1), t, nb);
    int const h4 = 2 * (t & 2);                                     // 4 * half
#pragma unroll
    for (int i = 0; i < 4; ++i) nb[i] = ~nb[i] >> h4;
    uint32_t const b = (sb + 96) & ~3u, shf = ((sb + 96) & 2u) * 8u;
    uint32_t const v0 = kr_lds32(b), v1 = kr_lds32(b + 4), v2 = kr_lds32(b + 8), v3 = kr_lds32(b + 12);
    uint32_t const a0 = __funnelshift_r(v0, v1, shf) >> h4, a1 = __funnelshift_r(v1, v2, shf) >> h4, a2 = __funnelshift_r(v2, v3, shf) >> h4;
    d = __half2float(__ushort_as_half(uint16_t(kr_lds16(sb + 108))));
    uint32_t const lo = (a0 & 0x0F0F0F0Fu) | ((a2 & 0x03030303u) << 4), hi = (a1 & 0x0F0F0F0Fu) | (((a2 >> 2) & 0x03030303u) << 4);
    uint32_t const p = uint32_t(t & 1);
    constexpr float up = kr_up<11>();
    s[0] = kr_scale(lo, p, up, -32.f);            s[1] = kr_scale(lo, p + 2, up * 0.25f, -32.f);
    s[2] = kr_scale(hi, p, up * 0.0625f, -32.f);  s[3] = kr_scale(hi, p + 2, up * 0.015625f, -32.f);
    sn[0] = __hmul2(s[0], __float2half2_rn(-4.f)); sn[1] = __hmul2(s[1], __float2half2_rn(-8.f));       // -4*sc / 2^j
    sn[2] = __hmul2(s[2], __float2half2_rn(-16.f)); sn[3] = __hmul2(s[3], __float2half2_rn(-32.f));
  }
  __device__ __forceinline__ void frag(int j, int wi, uint32_t (&a)[2]) const {
    uint32_t const m = 0x00030003u << (2 * j), hm = 0x00010001u << j;
    a[0] = h2_as_u32(__hfma2(kr_mask(nb[wi], hm), sn[j], __hmul2(kr_mask(q[wi], m), s[j])));
    a[1] = h2_as_u32(__hfma2(kr_mask(nb[wi] >> 8, hm), sn[j], __hmul2(kr_mask(q[wi] >> 8, m), s[j])));
  }
};

template <> struct KrRow<14> {                                      // Q6_K (2-byte aligned blocks)
  uint32_t q[2][4], hq[4];
  __half2 s[4], sh[4], sm[4];
  float d;
  __device__ __forceinline__ void load(uint32_t sb, int t) {
    uint32_t const c = 32 * (t & 2) + 16 * (t & 1);
    kr_run(sb + c, t, q[0]);
    kr_run(sb + c + 32, t, q[1]);
    kr_run(sb + 128 + 16 * t, t, hq);
    uint32_t const sa = sb + 192 + 4 * (t & 2), b = sa & ~3u, shf = (sa & 2u) * 8u;
    uint32_t const v0 = kr_lds32(b), v1 = kr_lds32(b + 4), v2 = kr_lds32(b + 8);
    uint32_t const lo = __funnelshift_r(v0, v1, shf) ^ 0x80808080u, hi = __funnelshift_r(v1, v2, shf) ^ 0x80808080u;
    d = __half2float(__ushort_as_half(uint16_t(kr_lds16(sb + 208))));
    uint32_t const p = uint32_t(t & 1);
    constexpr float up = kr_up<14>();
    __half2 const c0 = kr_scale(lo, p, up, -128.f), c1 = kr_scale(lo, p + 2, up, -128.f);
    __half2 const c2 = kr_scale(hi, p, up, -128.f), c3 = kr_scale(hi, p + 2, up, -128.f);
    __half2 const sixteenth = __float2half2_rn(0.0625f), off = __float2half2_rn(-0x1p-19f);             // -32 * 2^-24
    s[0] = c0; s[1] = c1; s[2] = __hmul2(c2, sixteenth); s[3] = __hmul2(c3, sixteenth);
    sh[0] = __hmul2(c0, __float2half2_rn(16.f)); sh[1] = __hmul2(c1, __float2half2_rn(4.f));            // 16*sc / 4^j
    sh[2] = c2; sh[3] = __hmul2(c3, __float2half2_rn(0.25f));
    sm[0] = __hmul2(c0, off); sm[1] = __hmul2(c1, off); sm[2] = __hmul2(c2, off); sm[3] = __hmul2(c3, off);
  }
  __device__ __forceinline__ void frag(int j, int wi, uint32_t (&a)[2]) const {
    uint32_t const w = q[j & 1][wi], m = (j & 2) ? 0x00F000F0u : 0x000F000Fu;
    a[0] = h2_as_u32(__hmul2(kr_mask(w, m), s[j]));
    a[1] = h2_as_u32(__hmul2(kr_mask(w >> 8, m), s[j]));
  }
  __device__ __forceinline__ void frag_high(int j, int wi, uint32_t (&a)[2]) const {
    uint32_t const m = 0x00030003u << (2 * j);
    a[0] = h2_as_u32(__hfma2(kr_mask(hq[wi], m), sh[j], sm[j]));
    a[1] = h2_as_u32(__hfma2(kr_mask(hq[wi] >> 8, m), sh[j], sm[j]));
  }
};

// Where field j, word wi of lane t sits in the superblock (first of its four consecutive elements), and its group.
template <int QT> __device__ __forceinline__ int kr_elem(int j, int wi, int t) {
  if constexpr (QT == 12 || QT == 13) return 32 * ((t & 2) + 4 * (j >> 1) + (j & 1)) + 16 * (t & 1) + 4 * wi;
  else return 64 * (t & 2) + 32 * j + 16 * (t & 1) + 4 * ((wi + t) & 3);
}
template <int QT> __device__ __forceinline__ int kr_group(int j, int t) {
  if constexpr (QT == 12 || QT == 13) return (t & 2) + 4 * (j >> 1) + (j & 1);
  else return 4 * (t & 2) + 2 * j + (t & 1);
}

// The segments of a CTA: runs of tiles of one (expert, eight-row group).
struct KrWalk {
  int u, u_end, e;
  int arow, nrows, t0, t1;
  __device__ __forceinline__ bool next(KrArgs const& a, int const* off, int const* cum) {
    if (u >= u_end) return false;
    int const gi = u / a.tiles;
    t0 = u - gi * a.tiles;
    t1 = min(min(a.tiles, t0 + (u_end - u)), t0 + a.round);
    u += t1 - t0;
    if (off) {
      while (cum[e] <= gi) ++e;                                     // cum: groups up to and with expert e
      int const first = off[e] + (gi - (e ? cum[e - 1] : 0)) * kKrCols;
      arow = first;
      nrows = min(kKrCols, off[e + 1] - first);
    } else {
      arow = gi * kKrCols;
      nrows = min(kKrCols, a.m_rows - arow);
    }
    return true;
  }
};

// Position in a ring of barriers: slot, phase parity of the current lap, and whether a lap is complete.
struct KrRing {
  unsigned i, phase;
  bool lap;
  __device__ __forceinline__ void step(int n) { if (++i == unsigned(n)) { i = 0; phase ^= 1u; lap = true; } }
};

struct KrBars { uint64_t full[kKrMaxStages], empty[kKrMaxStages], xfull[2], xempty[2], pfull[2], pempty[2], cfull; };

// One computing warp: its superblock of every tile of the CTA.
template <int QT, bool FINE>
__device__ __forceinline__ void kr_compute(KrArgs const& a, KrWalk wk, int const* offp, int const* cum, uint8_t* ring, uint8_t* xs, float* part,
                                           KrBars* bar, uint32_t stage_bytes, int warp, int lane, int k0) {
  constexpr int kBytes = kq::Fmt<QT>::kBytes;
  constexpr bool kHasMin = kq::Fmt<QT>::kHasMin;
  constexpr int kMin = QT == 10 ? 2 : 1;                            // pairs of sub-mins per lane and row
  constexpr int kChain = QT == 14 ? (FINE ? 2 : 8) : 4;             // fragments of a chain
  bool dead = false;
  int const g = lane >> 2, t = lane & 3;
  int const slot = warp / a.P, b = warp - slot * a.P;
  uint32_t const ring32 = smem_u32(ring) + uint32_t(slot * kKrTile + g) * a.pitch + b * kBytes;
  uint32_t const x32 = smem_u32(xs) + uint32_t(g) * a.xpitch + b * 512;
  float* const mypart = part + warp * kKrTile * kKrCols + g * kKrCols + 2 * t;
  uint32_t const row_step = uint32_t(a.bpr) * kBytes;               // low 32 bits are enough for the misalignment of a row
  KrRing ws{}, xr{}, pr{};
  bool first = a.xrows <= kKrDirectRows;
  while (!dead && wk.next(a, offp, cum)) {
    for (int p = 0; p < a.passes && !dead; ++p) {
      bool const active = k0 + p * a.P + b < a.bpr;
      uint32_t bf[16][2];
      bool const have = active && g < wk.nrows;
      if (first) {
        __half const* xg = a.x + (size_t(wk.arow + (have ? g : 0)) * a.bpr + (have ? k0 + b : 0)) * 256;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          uint2 v = make_uint2(0u, 0u);
          if (have) asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(xg + kr_elem<QT>(i >> 2, i & 3, t)));
          bf[i][0] = v.x; bf[i][1] = v.y;
        }
      } else {
        if (!mbar_wait_bounded(&bar->xfull[xr.i], xr.phase, a.status, kWaitStageTimeout)) { dead = true; break; }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          uint2 v = make_uint2(0u, 0u);
          if (have) v = kr_lds64(x32 + uint32_t(xr.i * a.xrows) * a.xpitch + 2 * kr_elem<QT>(i >> 2, i & 3, t));
          bf[i][0] = v.x; bf[i][1] = v.y;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar->xempty[xr.i]);
        xr.step(a.xbufs);
      }
      first = false;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        uint32_t const lo = bf[i][0], hi = bf[i][1];
        bf[i][0] = __byte_perm(lo, hi, 0x5410); bf[i][1] = __byte_perm(lo, hi, 0x7632);
      }
      uint32_t bs[3][kMin];                                         // group sums: B registers of the sub-min MMAs, three bf16 parts
      if constexpr (kHasMin) {
        float c4[4][4] = {};                                        // four chains: an MMA waits for the one before it
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          int const j = i & 3, grp = kr_group<QT>(j, t);
          uint32_t const lo = g == grp ? 0x3C003C00u : 0u, hi = g + 8 == grp ? 0x3C003C00u : 0u;
          kr_mma(c4[j], lo, hi, lo, hi, bf[j * 4 + (i >> 2)][0], bf[j * 4 + (i >> 2)][1]);
        }
        float c[4];                                                 // the chains are different groups: all but one are zero
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = (c4[0][i] + c4[1][i]) + (c4[2][i] + c4[3][i]);
        // row = group, column = activation row -> k index = group (2t, 2t+1 and, with 16 groups, 2t+8, 2t+9), column g
#pragma unroll
        for (int h = 0; h < kMin; ++h) {
          float v[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            int const src = 4 * (2 * t + i) + (g >> 1);
            float const e0 = __shfl_sync(0xffffffffu, c[2 * h], src), e1 = __shfl_sync(0xffffffffu, c[2 * h + 1], src);
            v[i] = (g & 1) ? e1 : e0;
          }
#pragma unroll
          for (int part = 0; part < 3; ++part) {
            bs[part][h] = __byte_perm(__float_as_uint(v[0]), __float_as_uint(v[1]), 0x7632);
            v[0] -= __uint_as_float(__float_as_uint(v[0]) & 0xFFFF0000u);
            v[1] -= __uint_as_float(__float_as_uint(v[1]) & 0xFFFF0000u);
          }
        }
      }
      uint32_t mis = 0, mis_step = 0;                               // rows of Q4_K and Q5_K are 16-byte aligned
      if constexpr (QT != 12 && QT != 13) {
        mis = uint32_t(reinterpret_cast<uintptr_t>(a.blocks)) + (uint32_t(a.offsets ? wk.e : 0) * uint32_t(a.n) + uint32_t((wk.t0 + slot) * kKrTile + g)) * row_step +
              uint32_t(k0 + p * a.P) * kBytes;
        mis_step = uint32_t(a.RS * kKrTile) * row_step;
      }
      for (int tb = wk.t0; tb < wk.t1; tb += a.RS, ws.step(a.stages), pr.step(2)) {
        if (!mbar_wait_bounded(&bar->full[ws.i], ws.phase, a.status, kWaitStageTimeout)) { dead = true; break; }
        bool const work = active && tb + slot < wk.t1;
        float2 o0 = make_float2(0.f, 0.f), o1 = o0;
        if (work) {
          uint32_t const base = ring32 + ws.i * stage_bytes;
          KrRow<QT> r0, r1;
          r0.load(base + (mis & 15u), t);
          r1.load(base + 8u * a.pitch + ((mis + 8u * row_step) & 15u), t);
          float cm[4] = {0.f, 0.f, 0.f, 0.f};                       // smallest part first
          if constexpr (QT == 10) {
#pragma unroll
            for (int part = 2; part >= 0; --part) kr_mma_bf16(cm, r0.mn[0], r1.mn[0], r0.mn[kMin - 1], r1.mn[kMin - 1], bs[part][0], bs[part][kMin - 1]);
          } else if constexpr (kHasMin) {
            kr_mma_bf16(cm, r0.mn[0], r1.mn[0], r0.mn[0], r1.mn[0], bs[2][0], bs[1][0]);
            kr_mma_bf16_k8(cm, r0.mn[0], r1.mn[0], bs[0][0]);
          }
          float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f}, p0[4], p1[4];   // even and odd fragments
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            uint32_t f0[2], f1[2];
            r0.frag(i >> 2, i & 3, f0);
            r1.frag(i >> 2, i & 3, f1);
            if constexpr (QT == 14 && !FINE) {                      // low nibbles and high bits apart
              kr_mma(s0, f0[0], f1[0], f0[1], f1[1], bf[i][0], bf[i][1]);
              r0.frag_high(i >> 2, i & 3, f0);
              r1.frag_high(i >> 2, i & 3, f1);
              kr_mma(s1, f0[0], f1[0], f0[1], f1[1], bf[i][0], bf[i][1]);
            } else {
              float (&p)[4] = (i & 1) ? p1 : p0;
              if ((i >> 1) % kChain == 0) kr_mma0(p, f0[0], f1[0], f0[1], f1[1], bf[i][0], bf[i][1]);
              else kr_mma(p, f0[0], f1[0], f0[1], f1[1], bf[i][0], bf[i][1]);
              if constexpr (QT == 14) {
                r0.frag_high(i >> 2, i & 3, f0);
                r1.frag_high(i >> 2, i & 3, f1);
                kr_mma(p, f0[0], f1[0], f0[1], f1[1], bf[i][0], bf[i][1]);
              }
              if ((i >> 1) % kChain == kChain - 1) {
                float (&s)[4] = (i & 1) ? s1 : s0;
#pragma unroll
                for (int j = 0; j < 4; ++j) s[j] = (i >> 1) < kChain ? p[j] : s[j] + p[j];
              }
            }
          }
          constexpr float down = 16777216.f / kr_up<QT>();
          float const d0 = r0.d * down, d1 = r1.d * down;
          o0.x = d0 * (s0[0] + s1[0]); o0.y = d0 * (s0[1] + s1[1]);
          o1.x = d1 * (s0[2] + s1[2]); o1.y = d1 * (s0[3] + s1[3]);
          if constexpr (kHasMin) {
            o0.x = fmaf(-r0.dmin, cm[0], o0.x); o0.y = fmaf(-r0.dmin, cm[1], o0.y);
            o1.x = fmaf(-r1.dmin, cm[2], o1.x); o1.y = fmaf(-r1.dmin, cm[3], o1.y);
          }
        }
        mis += mis_step;
        __syncwarp();                                               // every lane's reads of the stage are done
        if (lane == 0) mbar_arrive(&bar->empty[ws.i]);
        if (pr.lap && !mbar_wait_bounded(&bar->pempty[pr.i], pr.phase ^ 1u, a.status, kWaitStageTimeout)) { dead = true; break; }
        if (work) {
          float* const o = mypart + pr.i * kKrWarps * kKrTile * kKrCols;
          *reinterpret_cast<float2*>(o) = o0;
          *reinterpret_cast<float2*>(o + 8 * kKrCols) = o1;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar->pfull[pr.i]);
      }
    }
  }
}

// A ring stage of a tile at an end of the tensor [lo, hi) that is off a 16-byte boundary (rare, and kept out of the copy warp's loop).
__device__ __noinline__ void kr_copy_ends(uint8_t* stage, int pitch, uintptr_t b0, size_t step, int rows, unsigned len, uintptr_t lo, uintptr_t hi,
                                          uint64_t* full, int lane) {
  unsigned total = 0;
  for (int r = lane; r < rows; r += 32) {
    uintptr_t const b = b0 + size_t(r) * step;
    KrSpan const s = kr_span(b, len, lo, hi);
    uint8_t* const dst = stage + size_t(r) * pitch;
    total += unsigned(s.to - s.from);
    for (uintptr_t p = b; p < s.from; ++p) dst[p - s.first] = __ldg(reinterpret_cast<uint8_t const*>(p));
    for (uintptr_t p = s.to; p < b + len; ++p) dst[p - s.first] = __ldg(reinterpret_cast<uint8_t const*>(p));
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  total = __reduce_add_sync(0xffffffffu, total);                    // and the bytes are written before lane 0 arrives
  __syncwarp();
  if (lane == 0) mbar_expect_tx(full, total);
  __syncwarp();
  for (int r = lane; r < rows; r += 32) {
    KrSpan const s = kr_span(b0 + size_t(r) * step, len, lo, hi);
    bulk_g2s(stage + size_t(r) * pitch + (s.from - s.first), reinterpret_cast<void const*>(s.from), unsigned(s.to - s.from), full);
  }
}

// FINE: short chains for Q6_K (see "Rounding")
template <int QT, bool FINE>
__global__ void __launch_bounds__(kKrThreads, 1) kq_rows_kernel(KrArgs a) {
  constexpr int kBytes = kq::Fmt<QT>::kBytes;
  extern __shared__ __align__(128) uint8_t smem[];
  int const warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  int const active_warps = a.RS * a.P;
  // the CTAs of a cluster share their tiles and cut K: this one's superblocks are [k0, k0 + passes * P)
  int const rank = a.C > 1 ? int(blockIdx.x) % a.C : 0;
  int const k0 = rank * a.passes * a.P;
  bool const keep_sums = a.passes > 1 || a.C > 1;

  uint32_t const stage_bytes = uint32_t(a.RS) * kKrTile * a.pitch;
  uint8_t* ring = smem;
  uint8_t* xs = ring + a.stages * stage_bytes;                      // [xbufs][xrows][xpitch]
  float* part = reinterpret_cast<float*>(xs + size_t(a.xbufs) * a.xrows * a.xpitch);      // [2][16][16 rows][8 cols]
  float* acc = part + 2 * kKrWarps * kKrTile * kKrCols;             // [2][round][16][8], several passes or CTAs only
  unsigned const acc_floats = keep_sums ? unsigned(a.round) * kKrTile * kKrCols : 0u;
  KrBars* bar = reinterpret_cast<KrBars*>(acc + 2 * acc_floats);
  int* off = reinterpret_cast<int*>(bar + 1);                       // [experts+1], then cum [experts]
  int* cum = off + a.experts + 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) { mbar_init(&bar->full[s], 1); mbar_init(&bar->empty[s], active_warps); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar->xfull[s], 1); mbar_init(&bar->xempty[s], active_warps);
      mbar_init(&bar->pfull[s], active_warps); mbar_init(&bar->pempty[s], 1);
    }
    mbar_init(&bar->cfull, a.C);
    mbar_init_fence();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();
  if (a.C > 1) {                                                    // nobody arrives on a barrier that is not there yet
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  // Under programmatic dependent launch nothing of the activations, the offsets or the output is touched before this.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int groups = kr_groups(a.m_rows);
  if (a.offsets) {
    // The offsets may not have been checked: they are settled first, so that no later index depends on what else they hold.
    for (int i = threadIdx.x; i <= a.experts; i += kKrThreads) off[i] = a.offsets[i];
    __syncthreads();
    if (warp == 0) {
      int top = 0;
      for (int base = 0; base <= a.experts; base += 32) {           // running maximum of the clamped offsets
        int const i = base + lane;
        int v = kr_settle(0, i <= a.experts ? off[i] : 0, a.m_rows);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { int const p = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v = kr_settle(p, v, a.m_rows); }
        v = kr_settle(top, v, a.m_rows);
        if (i <= a.experts) off[i] = v;
        top = __shfl_sync(0xffffffffu, v, 31);
      }
      __syncwarp();
      int carry = 0;                                                // inclusive scan of the experts' group counts
      for (int base = 0; base < a.experts; base += 32) {
        int const i = base + lane;
        int v = i < a.experts ? kr_groups(off[i + 1] - off[i]) : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { int const p = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += p; }
        v += carry;
        if (i < a.experts) cum[i] = v;
        carry = __shfl_sync(0xffffffffu, v, 31);
      }
    }
  }
  __syncthreads();
  if (a.offsets) groups = cum[a.experts - 1];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  long long const units = (long long)groups * a.tiles;
  unsigned const part_i = blockIdx.x / a.C, part_n = gridDim.x / a.C;
  KrWalk wk{};
  wk.u = kr_cut(units, part_i, part_n);
  wk.u_end = kr_cut(units, part_i + 1, part_n);
  int const* offp = a.offsets ? off : nullptr;
  bool dead = false;

  if (warp == kKrWarps) {
    // ---- copies ---------------------------------------------------------------------------------------------------------
    KrRing ws{}, xr{};
    uintptr_t const lo = reinterpret_cast<uintptr_t>(a.blocks), hi = lo + size_t(a.offsets ? a.experts : 1) * a.n * a.bpr * kBytes;
    bool const odd_ends = ((lo | hi) & 15u) != 0;
    bool first = a.xrows <= kKrDirectRows;                          // the computing warps load these activations themselves
    while (!dead && wk.next(a, offp, cum)) {
      for (int p = 0; p < a.passes && !dead; ++p) {
        int const sb0 = k0 + p * a.P, nb = max(0, min(a.P, a.bpr - sb0));
        if (!first) {
          if (xr.lap && !mbar_wait_bounded(&bar->xempty[xr.i], xr.phase ^ 1u, a.status, kWaitStageTimeout)) { dead = true; break; }
          if (lane == 0) mbar_expect_tx(&bar->xfull[xr.i], unsigned(wk.nrows * nb) * 512u);
          __syncwarp();
          if (lane < wk.nrows && nb)
            bulk_g2s(xs + size_t(xr.i * a.xrows + lane) * a.xpitch, a.x + (size_t(wk.arow + lane) * a.bpr + sb0) * 256, unsigned(nb) * 512u, &bar->xfull[xr.i]);
          xr.step(a.xbufs);
        }
        first = false;
        unsigned const len = unsigned(nb) * kBytes;
        size_t const step = size_t(a.bpr) * kBytes;
        uint8_t const* src0 = a.blocks + ((size_t(a.offsets ? wk.e : 0) * a.n + size_t(wk.t0) * kKrTile) * a.bpr + size_t(sb0)) * kBytes;
        for (int tb = wk.t0; tb < wk.t1; tb += a.RS, ws.step(a.stages), src0 += size_t(a.RS * kKrTile) * step) {
          if (ws.lap && !mbar_wait_bounded(&bar->empty[ws.i], ws.phase ^ 1u, a.status, kWaitStageTimeout)) { dead = true; break; }
          int const rows = nb ? min(min(a.RS, wk.t1 - tb) * kKrTile, a.n - tb * kKrTile) : 0;
          uint8_t* const stage = ring + ws.i * stage_bytes;
          // a tensor that begins or ends inside a 16-byte unit: its first and last tiles are copied with that in mind
          if (QT != 12 && QT != 13 && odd_ends && (tb == 0 || tb + a.RS >= a.tiles)) {
            kr_copy_ends(stage, a.pitch, reinterpret_cast<uintptr_t>(src0), step, rows, len, lo, hi, &bar->full[ws.i], lane);
            continue;
          }
          auto span = [&](int r, uint8_t const*& from) -> unsigned {    // the 16-byte units that hold row r's segment
            uintptr_t const b = reinterpret_cast<uintptr_t>(src0 + size_t(r) * step);
            from = reinterpret_cast<uint8_t const*>(b & ~uintptr_t(15));
            return unsigned(((b + len + 15) & ~uintptr_t(15)) - (b & ~uintptr_t(15)));
          };
          unsigned total = 0;
          uint8_t const* from;
          for (int r = lane; r < rows; r += 32) total += span(r, from);
          total = __reduce_add_sync(0xffffffffu, total);
          if (lane == 0) mbar_expect_tx(&bar->full[ws.i], total);
          __syncwarp();
          for (int r = lane; r < rows; r += 32) {
            unsigned const bytes = span(r, from);
            bulk_g2s(stage + size_t(r) * a.pitch, from, bytes, &bar->full[ws.i]);
          }
        }
      }
    }
    if (dead) {                                                     // let what is in flight land before the memory is handed on
      // (a slot below the current one was filled in this lap, the others in the lap before)
      for (unsigned i = 0; i < unsigned(a.stages); ++i)
        if (ws.lap || i < ws.i) (void)mbar_wait_bounded(&bar->full[i], i < ws.i ? ws.phase : ws.phase ^ 1u, nullptr, 0, 250000000ull);
      for (unsigned i = 0; i < unsigned(a.xbufs); ++i)
        if (xr.lap || i < xr.i) (void)mbar_wait_bounded(&bar->xfull[i], i < xr.i ? xr.phase : xr.phase ^ 1u, nullptr, 0, 250000000ull);
    }
  } else if (warp > kKrWarps) {
    // ---- K slices of a tile, added in warp order, then in CTA order ---------------------------------------------------------
    KrRing pr{};
    unsigned seg = 0;
    auto store = [&](int tile, float4 v) {
      int const row = tile * kKrTile + (lane >> 1), col = (lane & 1) * 4;
      if (row < a.n) {
        float* o = a.out + size_t(wk.arow + col) * a.n + row;
        if (col < wk.nrows) o[0] = v.x;
        if (col + 1 < wk.nrows) o[a.n] = v.y;
        if (col + 2 < wk.nrows) o[2 * size_t(a.n)] = v.z;
        if (col + 3 < wk.nrows) o[3 * size_t(a.n)] = v.w;
      }
    };
    while (!dead && wk.next(a, offp, cum)) {
      float* const seg_acc = acc + (seg & 1u) * acc_floats;
      for (int p = 0; p < a.passes && !dead; ++p) {
        int const nb = max(0, min(a.P, a.bpr - k0 - p * a.P));
        for (int tb = wk.t0; tb < wk.t1; tb += a.RS, pr.step(2)) {
          if (!mbar_wait_bounded(&bar->pfull[pr.i], pr.phase, a.status, kWaitStageTimeout)) { dead = true; break; }
          int const nt = min(a.RS, wk.t1 - tb);
          for (int sl = 0; sl < nt; ++sl) {
            float4 const* src = reinterpret_cast<float4 const*>(part + (pr.i * kKrWarps + sl * a.P) * kKrTile * kKrCols) + lane;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f), u = v;      // even and odd superblocks
            auto add = [](float4& to, float4 o) { to.x += o.x; to.y += o.y; to.z += o.z; to.w += o.w; };
#pragma unroll 8
            for (int b = 0; b + 1 < nb; b += 2) {
              add(v, src[b * (kKrTile * kKrCols / 4)]);
              add(u, src[(b + 1) * (kKrTile * kKrCols / 4)]);
            }
            if (nb & 1) add(v, src[(nb - 1) * (kKrTile * kKrCols / 4)]);
            add(v, u);
            if (keep_sums) {
              float4* keep = reinterpret_cast<float4*>(seg_acc + (tb + sl - wk.t0) * kKrTile * kKrCols) + lane;
              if (p > 0) { float4 const o = *keep; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
              if (p + 1 < a.passes || a.C > 1) { *keep = v; continue; }
            }
            store(tb + sl, v);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar->pempty[pr.i]);
        }
      }
      if (a.C > 1 && !dead) {
        // every CTA of the cluster has its share of the segment: each adds a part of the tiles.  The sums are kept in two
        // buffers by turns, so a CTA that runs ahead waits for this segment's readers before it overwrites what they read.
        __syncwarp();
        if (lane < a.C)
          asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\tmbarrier.arrive.release.cluster.shared::cluster.b64 _, [r];\n\t}"
                       ::"r"(smem_u32(&bar->cfull)), "r"(lane) : "memory");
        if (!mbar_wait_bounded(&bar->cfull, seg & 1u, a.status, kWaitStageTimeout)) { dead = true; break; }
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        for (int i = rank; i < wk.t1 - wk.t0; i += a.C) {
          uint32_t const at = smem_u32(seg_acc + i * kKrTile * kKrCols) + 16u * lane;
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int c = 0; c < a.C; ++c) {
            float4 o;
            asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %4, %5;\n\tld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [r];\n\t}"
                         : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(at), "r"(c) : "memory");
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
          }
          store(wk.t0 + i, v);
        }
        __syncwarp();
      }
      ++seg;
    }
  } else if (warp < active_warps) {
    kr_compute<QT, FINE>(a, wk, offp, cum, ring, xs, part, bar, stage_bytes, warp, lane, k0);
  }
  if (a.C > 1) {                                                    // a CTA's sums are read by the others until here
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

struct KrPlan { int passes, P, RS, C, pitch, xpitch, stages, xbufs, round, slots, ok; size_t smem; };

void kr_launch_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&at)[2], KrPlan const& p, unsigned grid, cudaStream_t stream) {
  static bool const no_pdl = std::getenv("QUACTLIZE_B200_NO_PDL") != nullptr;
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(kKrThreads); cfg.dynamicSmemBytes = p.smem; cfg.stream = stream;
  int na = 0;
  if (p.C > 1) { at[na].id = cudaLaunchAttributeClusterDimension; at[na].val.clusterDim.x = unsigned(p.C); at[na].val.clusterDim.y = at[na].val.clusterDim.z = 1; ++na; }
  if (!no_pdl) { at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[na].val.programmaticStreamSerializationAllowed = 1; ++na; }
  cfg.attrs = at; cfg.numAttrs = unsigned(na);
}

// Shared memory of a split; false where it does not fit two ring stages.
template <int QT>
bool kr_layout(KrPlan& p, int xrows, int experts) {
  constexpr int kBytes = kq::Fmt<QT>::kBytes;
  constexpr bool aligned = QT == 12 || QT == 13;
  int pitch = (p.P * kBytes + (aligned ? 0 : 15 + 4) + 15) / 16 * 16;
  while (pitch % 128 != (aligned ? 64 : 16)) pitch += 16;
  p.pitch = pitch;
  p.xpitch = p.P * 512 + 16;
  bool const keep = p.passes > 1 || p.C > 1;
  p.round = keep ? kKrAccTiles / p.RS * p.RS : 1 << 28;
  size_t const tile = size_t(kKrTile) * kKrCols * 4;
  size_t const fixed = 2 * kKrWarps * tile + (keep ? 2 * p.round * tile : 0) + sizeof(KrBars) + (size_t(2) * experts + 1) * 4;
  size_t const stage = size_t(p.RS) * kKrTile * p.pitch, xbuf = size_t(xrows) * p.xpitch;
  p.xbufs = p.passes > 1 && fixed + 2 * xbuf + 4 * stage <= kKrSmem ? 2 : 1;
  p.stages = fixed + p.xbufs * xbuf < kKrSmem ? int(std::min<size_t>(kKrMaxStages, (kKrSmem - fixed - p.xbufs * xbuf) / stage)) : 0;
  p.smem = fixed + p.xbufs * xbuf + p.stages * stage;
  return p.stages >= 2;
}

// Clusters of C CTAs that the GPCs hold at the same time (the kernel takes an SM per CTA whatever its shared memory); 0: none.
template <int QT, bool FINE>
int kr_resident(int C) {
  if (C == 1) return rt_sm_count();
  KrPlan p{};
  p.C = C; p.smem = kKrSmem;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  int const most = rt_sm_count() / C;
  kr_launch_config(cfg, at, p, unsigned(most * C), nullptr);
  int resident = 0;
  if (cudaOccupancyMaxActiveClusters(&resident, kq_rows_kernel<QT, FINE>, &cfg) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  return std::min(most, resident);
}

// `units`: tiles of the launch (ragged: those of a router that spreads its rows).  Plans are kept per shape.
template <int QT, bool FINE>
KrPlan kr_plan(int bpr, int units, int xrows, int experts) {
  constexpr int kSplits[3] = {1, 2, 4};
  units = std::min(units, 64 * rt_sm_count());                      // beyond that the split no longer depends on it
  struct Key { int bpr, units, x, e, dev; bool operator<(Key const& o) const {
    return bpr != o.bpr ? bpr < o.bpr : units != o.units ? units < o.units : x != o.x ? x < o.x : e != o.e ? e < o.e : dev < o.dev; } };
  struct Slots { int n[3]; };
  static std::map<Key, KrPlan> plans;
  static std::map<int, Slots> resident;                             // per device
  static std::mutex mu;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  Key const key{bpr, units, xrows, experts, dev};
  auto it = plans.find(key);
  if (it != plans.end()) return it->second;
  auto rs = resident.find(dev);
  if (rs == resident.end()) {
    Slots v{};
    if (cudaFuncSetAttribute(kq_rows_kernel<QT, FINE>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kKrSmem)) == cudaSuccess)
      for (int i = 0; i < 3; ++i) v.n[i] = kr_resident<QT, FINE>(kSplits[i]);
    else
      (void)cudaGetLastError();
    rs = resident.emplace(dev, v).first;
  }
  if (plans.size() > 4096) plans.clear();
  KrPlan bestp{};
  double best = 1e30;
  for (int i = 0; i < 3; ++i) {
    int const C = kSplits[i], slots = rs->second.n[i];
    if (slots <= 0) continue;
    int const per_cta = (bpr + C - 1) / C, least = (per_cta + kKrWarps - 1) / kKrWarps;
    for (int passes = least; passes <= std::min(per_cta, least + 2); ++passes) {
      KrPlan p{};
      p.C = C; p.passes = passes; p.slots = slots;
      p.P = (per_cta + passes - 1) / passes; p.RS = kKrWarps / p.P;
      if (!kr_layout<QT>(p, xrows, experts)) continue;
      // Microseconds on 4096-deep Q4_K rows: a stage costs a latency and its warps' share of the issue slots, a pass the
      // reload of the activations, a cluster the exchange of its sums.  Rounds are counted over the clusters that are resident
      // (74 of two CTAs, but 33 of four on 148 SMs): 14336 -> 8192, Q4_K 2 rows 26.2 us as fours, 24.4 as twos, 25.8 whole, and the
      // other way round where there are few tiles, 14336 -> 4096 15.4, 16.0, 15.9.
      int const rounds = ((units + slots - 1) / slots + p.RS - 1) / p.RS * passes;
      double const cost = rounds * (0.4 + 0.8 * p.RS * p.P / kKrWarps) + 0.9 * passes + (C > 1 ? 1.0 : 0.0);
      if (cost < best - 1e-9) { best = cost; bestp = p; bestp.ok = 1; }
    }
  }
  return plans.emplace(key, bestp).first->second;
}

template <int QT, bool FINE = false>
bool launch(KrArgs a, cudaStream_t stream) {
  a.tiles = (a.n + kKrTile - 1) / kKrTile;
  a.xrows = std::min(kKrCols, a.m_rows);
  int const most = a.offsets ? kr_most_groups(a.m_rows, a.experts) : kr_groups(a.m_rows);
  if ((long long)most * a.tiles > kKrMaxUnits) return false;
  // a router that spreads r rows over E experts touches about r of them while r is small against E
  int const likely = a.offsets ? std::max(1, std::min(most, int((long long)a.m_rows * a.experts / (a.m_rows + a.experts)))) : most;
  KrPlan const p = kr_plan<QT, FINE>(a.bpr, likely * a.tiles, a.xrows, a.experts);
  if (!p.ok) return false;
  a.passes = p.passes; a.P = p.P; a.RS = p.RS; a.C = p.C; a.pitch = p.pitch; a.xpitch = p.xpitch; a.stages = p.stages; a.xbufs = p.xbufs; a.round = p.round;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  kr_launch_config(cfg, at, p, unsigned(std::min(p.slots, most * a.tiles) * p.C), stream);
  if (cudaLaunchKernelEx(&cfg, kq_rows_kernel<QT, FINE>, a) != cudaSuccess) { (void)cudaGetLastError(); return false; }
  return true;
}

}  // namespace

// Enqueue; false when the problem is outside this kernel's envelope (the caller then uses another kernel).
bool enqueue_kq_rows(uint8_t const* blocks, __half const* x, float* out, int const* offsets, int n, int bpr, int experts, int rows,
                     int qtype, unsigned int* status, cudaStream_t stream) {
  if (n <= 0 || bpr <= 0 || rows <= 0 || !status || (offsets && experts > kKrMaxExperts)) return false;
  uintptr_t const need = qtype == 12 || qtype == 13 ? 15 : qtype == 10 ? 3 : 1;
  if ((reinterpret_cast<uintptr_t>(blocks) & need) || (reinterpret_cast<uintptr_t>(x) & 15)) return false;
  KrArgs a{};
  a.blocks = blocks; a.x = x; a.out = out; a.offsets = offsets; a.n = n; a.bpr = bpr; a.experts = offsets ? experts : 0; a.m_rows = rows; a.status = status;
  switch (qtype) {
    case 10: return launch<10>(a, stream);
    case 11: return launch<11>(a, stream);
    case 12: return launch<12>(a, stream);
    case 13: return launch<13>(a, stream);
    case 14: return (reinterpret_cast<uintptr_t>(blocks) | size_t(bpr) * 210) % 16 ? launch<14, true>(a, stream) : launch<14>(a, stream);
    default: return false;
  }
}

}  // namespace qb
