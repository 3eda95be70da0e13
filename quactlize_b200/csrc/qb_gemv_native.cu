// Decode GEMV over RAW GGUF k-quant blocks (the checkpoint's own bytes; nothing is materialised).
//
//   out[t, r] = sum_k x[t, k] * W[r, k],   W from blocks [E][n][k/256][block_bytes] row-major by output row,
//   x fp16 [rows, k] (dense: shared by all rows; grouped: gathered in expert order with cumulative offsets),
//   out fp32.
//
// Replaces the reference kernel vecdot_rows_kernel (quactlize/include/gguf_vecdot.hpp:604-760) and its launch policy
// (quactlize/csrc/device/ppu_backend.cu:52-131).  The arithmetic identity is the reference's
// (gguf_vecdot.hpp:12-19): sum_i W_i x_i = sum_g [ dl_g * sum(q x) - ml_g * sum(x) ], but group sums are carried to
// fp32 after at most 16 fp16 products instead of accumulating the whole row in fp16.
//
// This file holds the launch policy and the plain kernel (any format, any alignment, blocks read through L1, one warp per
// output row); the kernels that stream the weights through shared memory are in qb_gemv_q4k.cu and qb_gemv_kquant1.cu (one
// activation row), qb_gemv_q4k_rows.cu and qb_gemv_kqrows.cu (several).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "qb_device.cuh"
#include "qb_internal.hpp"
#include "qb_kquant.cuh"
#include "qb_runtime.hpp"

namespace qb {

struct NativeArgs {
  uint8_t const* blocks;
  __half const* x;
  float* out;
  int const* offsets;     // cumulative [experts+1] (grouped) or nullptr (dense)
  int n, bpr, experts, m_rows, mtiles;
  int per_row_x;          // row r has its own activation slice (the per-block vecdot contract)
  unsigned int* status;
};

// ------------------------------------------------------------------------------------------------------------------
// Any k-quant, any alignment: one warp per output row, lanes stride over (block, group) items.

template <int QT, int M>
__global__ void __launch_bounds__(256) kquant_gemv_generic_kernel(NativeArgs a) {
  using F = kq::Fmt<QT>;
  constexpr int G = F::kGroups, GS = 256 / G;
  int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int const row = blockIdx.x * (blockDim.x >> 5) + warp;
  int e = 0, mt = blockIdx.y, row_base, mvalid;
  if (a.offsets) {
    e = blockIdx.y / a.mtiles; mt = blockIdx.y % a.mtiles;
    int const r0 = a.offsets[e], r1 = a.offsets[e + 1];
    row_base = r0 + mt * M; mvalid = min(M, r1 - row_base);
  } else {
    row_base = mt * M; mvalid = min(M, a.m_rows - row_base);
  }
  if (mvalid <= 0 || row >= a.n) return;
  int const k = a.bpr * 256;
  uint8_t const* rb = a.blocks + (size_t(e) * a.n + row) * a.bpr * F::kBytes;
  __half const* xb = a.per_row_x ? a.x + size_t(row) * k : a.x + size_t(row_base) * k;
  float acc[M];
#pragma unroll
  for (int m = 0; m < M; ++m) acc[m] = 0.f;
  for (int it = lane; it < a.bpr * G; it += 32) {
    int const b = it / G, g = it % G;
    uint8_t const* blk = rb + size_t(b) * F::kBytes;
    float const d = __half2float(__ushort_as_half(kq::load_u16(blk + F::kD)));
    float dmin = 0.f;
    if constexpr (F::kHasMin) dmin = __half2float(__ushort_as_half(kq::load_u16(blk + F::kDmin)));
    int sc, mn;
    kq::scale_min<QT>(blk + F::kScaleOff, g, sc, mn);
    float const dl = d * float(sc), ml = dmin * float(mn);
    float sqx[M], sxx[M];
#pragma unroll
    for (int m = 0; m < M; ++m) { sqx[m] = 0.f; sxx[m] = 0.f; }
    for (int j = 0; j < GS; ++j) {
      float const q = float(kq::code<QT>(blk, g, j));
#pragma unroll
      for (int m = 0; m < M; ++m) {
        if (m < mvalid) {
          float const xv = __half2float(xb[size_t(m) * k + b * 256 + g * GS + j]);
          sqx[m] = fmaf(q, xv, sqx[m]);
          sxx[m] += xv;
        }
      }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) acc[m] += dl * sqx[m] - ml * sxx[m];
  }
#pragma unroll
  for (int m = 0; m < M; ++m) {
    float const t = warp_sum(acc[m]);
    if (lane == 0 && m < mvalid) {
      if (a.per_row_x) a.out[row] = t; else a.out[size_t(row_base + m) * a.n + row] = t;
    }
  }
}

// ------------------------------------------------------------------------------------------------------------------
// host launch policy

namespace {

template <int QT, int M>
void launch_generic(NativeArgs const& a, int gy, cudaStream_t stream) {
  kquant_gemv_generic_kernel<QT, M><<<dim3((a.n + 7) / 8, gy), 256, 0, stream>>>(a);
}

template <int M>
void launch_generic_qt(int qtype, NativeArgs const& a, int gy, cudaStream_t stream) {
  switch (qtype) {
    case 10: launch_generic<10, M>(a, gy, stream); break;
    case 11: launch_generic<11, M>(a, gy, stream); break;
    case 12: launch_generic<12, M>(a, gy, stream); break;
    case 13: launch_generic<13, M>(a, gy, stream); break;
    default: launch_generic<14, M>(a, gy, stream); break;
  }
}

}  // namespace

// Enqueue a raw-block GEMV.  max_rows bounds the activation rows of any expert (dense: the row count).
// force_generic selects the simple kernel (used by tests to cross-check the two implementations).
int enqueue_native_gemv(uint8_t const* blocks, __half const* x, float* out, int const* offsets,
                        int n, int bpr, int experts, int m_rows, int max_rows, int qtype, bool per_row_x,
                        bool force_generic, cudaStream_t stream) {
  NativeArgs a{};
  a.blocks = blocks; a.x = x; a.out = out; a.offsets = offsets;
  a.n = n; a.bpr = bpr; a.experts = experts > 0 ? experts : 1; a.m_rows = m_rows;
  a.per_row_x = per_row_x ? 1 : 0;
  a.status = rt_device_status_ptr();
  int const rows_hint = offsets ? max_rows : m_rows;
  if (!per_row_x && !force_generic && a.status) {
    bool const aligned = (reinterpret_cast<uintptr_t>(blocks) % 16 == 0) && (reinterpret_cast<uintptr_t>(x) % 16 == 0);
    int const sms = rt_sm_count(), tiles = (n + 15) / 16;
    // One activation row per weight pass (a further row reads the weights from L2) against one pass for up to eight rows,
    // us on 4096-deep rows.  One row: 8.3-12 against 13-19 at n = 14336.
    //   two rows, few output rows: Q5_K n = 2400 6.6 against 7.3, n = 4800 9.3 against 9.3; a 2048-deep Q6_K 8.0 against 6.5
    //   Q2_K, the fewest bytes: 13.3 against 14.6 for two rows also at n = 14336
    //   three rows: Q5_K n = 1024 5.2 against 5.9, n = 2400 7.9 against 7.3
    //   14336-deep rows: two rows Q5_K n = 2048 12.7 against 11.9, three rows Q6_K n = 1024 12.0 against 9.7 (n = 1024, 8192-deep, 7.4
    //   against 8.1); Q2_K, two rows, n = 4096 15.3 against 17.6
    // Q4_K keeps fp32 sums from two rows up (relative error 5e-4 with the fp16 sums of the one-row kernel, 1e-7 without), at
    // 6.2 against 5.1 us for two rows of 8192, n = 1024.
    // Ragged launches always share: their offsets need not have been checked there, the call then has one kernel whatever the
    // type of its activations and its offsets, and sums stay fp32.  At most two rows per expert, one row per pass against it:
    // 2048-deep Q4_K, 12 rows of 32 experts, n = 8192 45.8 against 33.5, 64 rows of 128 experts, n = 1536 66.5 against 34.4; 4096-deep
    // 46.6 against 46.5, and 6 rows of 8 experts, n = 14336 39 against 45.
    bool const few = (m_rows == 2 && (qtype == 10 || (bpr <= 32 && tiles <= sms))) || (m_rows == 3 && bpr <= 32 && 2 * tiles <= sms);
    bool const one_row = !offsets && (m_rows == 1 || (qtype != 12 && bpr >= 16 && few));
    if (qtype == 12 && !offsets && m_rows >= 2 && m_rows <= 4 && bpr <= 16 && tiles <= 3 * sms) {
      // two to four Q4_K rows, few tiles per SM: no copy and reducing warps to start and drain (2 rows, n = 2400 5.2 against 6.0 us;
      // 4 rows, n = 7000 7.4 against 8.6; 2 rows, n = 14336 13.2 against 12.2)
      if (enqueue_q4k_rows(blocks, x, out, n, bpr, m_rows, a.status, stream)) return 0;
    }
    if (one_row && aligned) {
      if (qtype == 12 ? enqueue_q4k_gemv1(blocks, x, out, n, bpr, m_rows, a.status, stream)
                      : enqueue_kquant_gemv1(blocks, x, out, n, bpr, m_rows, qtype, a.status, stream)) return 0;
    }
    // Everything else, rows off a 16-byte boundary among it (K % 2048 != 0 for Q3_K and Q6_K, K % 1024 != 0 for Q2_K), which
    // the plain kernel took 67-141 us for at 14336 x 4096.
    if (enqueue_kq_rows(blocks, x, out, offsets, n, bpr, a.experts, m_rows, qtype, a.status, stream)) return 0;
  }
  if (per_row_x) {
    a.mtiles = 1;
    launch_generic_qt<1>(qtype, a, 1, stream);
    return 0;
  }
  int const mt = rows_hint >= 2 ? 4 : 1;
  a.mtiles = (rows_hint + mt - 1) / mt;
  int const gy = (offsets ? a.experts : 1) * a.mtiles;
  if (mt == 1) launch_generic_qt<1>(qtype, a, gy, stream); else launch_generic_qt<4>(qtype, a, gy, stream);
  return 0;
}

}  // namespace qb
