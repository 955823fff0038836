// tiled.cu -- shared-memory tiled gathers for the per-step kernels.
//
// The untiled gathers (force.cu) issue ten to thirteen scattered loads per
// neighbour entry and run at the L1 throughput limit with HBM far from busy.
// Here nodes are renumbered in bin-cell order (spatially compact), rows are
// grouped into tiles of R consecutive nodes, and each tile's neighbour set
// (the union of its rows, "J-set") is listed once.  Every neighbour entry
// then carries its gradient and a 16-bit tile-local index in one 16-byte
// (float) or 26-byte (double) record, laid out in slices of 8 rows so that a
// warp's loads are contiguous (build_slices), and the neighbour data the tile needs
// -- (u_tot, du) for the deformation gradient, T_i for the force -- is staged
// in shared memory once per tile:
//   k_defgrad_t  G0 = sum_J (du_J - du_i) (x) g + du_i (x) sum g, and on FULL
//                steps F - I likewise from u (on the others F advances by G0)
//   k_force_t    f_J = sum_i T_i g^T_iJ, then the corrector / predictor
// The summation order is fixed by the list order, so results are
// deterministic, and identical in exact arithmetic to force.cu's.
#include "mega_internal.cuh"
#include "stress.cuh"
#include "tiled.cuh"
#include "bulk.cuh"

namespace mega {
namespace {

// Launch variants of the two gathers (picked per context by the autotuner):
// KG lanes per row / column (4, 8 or 16), KU packed records in flight per
// lane (1, 2 or 4).  A block serves one tile of R rows with R * KG threads.
template <int KG>
__device__ __forceinline__ unsigned group_mask() {
  return ((1u << KG) - 1u) << (threadIdx.x & (32 - KG));
}

__device__ __forceinline__ unsigned hash_u32(unsigned x) {
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
  return x;
}

// Block per tile: list the distinct neighbours of the tile's rows, sort them,
// and give each entry its rank in that list.  HS hash slots in shared memory;
// a tile with more than jmax distinct neighbours reports overflow.
template <int HS>
__global__ void __launch_bounds__(256) k_build_tiles(int32_t n, int32_t R, const int64_t* __restrict__ ptr,
                                                     const int32_t* __restrict__ idx, int32_t jmax,
                                                     int32_t* __restrict__ jset, int32_t* __restrict__ jcnt,
                                                     uint16_t* __restrict__ lidx, int16_t* __restrict__ slot_tmp,
                                                     int32_t* __restrict__ overflow) {
  __shared__ int32_t keys[HS];
  __shared__ int16_t rank[HS];
  __shared__ int32_t sk[HS / 2];
  __shared__ int32_t wsum[8];
  __shared__ int32_t s_total, s_full;
  const int tid = threadIdx.x;
  const int64_t t = blockIdx.x;
  const int64_t r0 = t * R, r1 = min((int64_t)n, r0 + R);
  const int64_t p0 = ptr[r0], p1 = ptr[r1];
  for (int s = tid; s < HS; s += blockDim.x) keys[s] = -1;
  if (tid == 0) s_full = 0;
  __syncthreads();
  for (int64_t p = p0 + tid; p < p1; p += blockDim.x) {
    const int32_t j = idx[p];
    unsigned h = hash_u32((unsigned)j) & (HS - 1);
    int16_t slot = -1;
    for (int probe = 0; probe < HS; ++probe) {  // bounded: a full table stops
      const int32_t prev = atomicCAS(&keys[h], -1, j);
      if (prev == -1 || prev == j) { slot = (int16_t)h; break; }
      h = (h + 1) & (HS - 1);
    }
    if (slot < 0) s_full = 1;
    slot_tmp[p] = slot;
  }
  __syncthreads();
  // compaction of the occupied slots: each thread owns HS/256 consecutive slots
  constexpr int PER = HS / 256;
  int cnt = 0;
  for (int k = 0; k < PER; ++k) cnt += (keys[tid * PER + k] != -1);
  int x = cnt;
  const int lane = tid & 31, wid = tid >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[wid] = x;
  __syncthreads();
  if (tid == 0) {
    int a = 0;
    for (int w = 0; w < 8; ++w) { const int v = wsum[w]; wsum[w] = a; a += v; }
    s_total = a;
  }
  __syncthreads();
  const int total = s_total;
  if (total > jmax || s_full) {  // the whole block leaves together
    if (tid == 0) {
      jcnt[t] = total;
      atomicMax(overflow, s_full ? HS : total);
    }
    return;
  }
  int pos = wsum[wid] + x - cnt;
  for (int k = 0; k < PER; ++k) {
    const int32_t key = keys[tid * PER + k];
    if (key != -1) sk[pos++] = key;
  }
  int np2 = 1;
  while (np2 < total) np2 <<= 1;
  for (int s = total + tid; s < np2; s += blockDim.x) sk[s] = INT32_MAX;
  __syncthreads();
  // bitonic sort of sk[0..np2)
  for (int k = 2; k <= np2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < np2; i += blockDim.x) {
        const int l = i ^ j;
        if (l > i) {
          const int32_t a = sk[i], b = sk[l];
          const bool up = (i & k) == 0;
          if ((a > b) == up) { sk[i] = b; sk[l] = a; }
        }
      }
      __syncthreads();
    }
  // rank of each slot = position of its key in the sorted list
  for (int r = tid; r < total; r += blockDim.x) {
    const int32_t key = sk[r];
    unsigned h = hash_u32((unsigned)key) & (HS - 1);
    for (int probe = 0; probe < HS; ++probe) {
      if (keys[h] == key) { rank[h] = (int16_t)r; break; }
      h = (h + 1) & (HS - 1);
    }
    jset[t * (int64_t)jmax + r] = key;
  }
  if (tid == 0) jcnt[t] = total;
  __syncthreads();
  for (int64_t p = p0 + tid; p < p1; p += blockDim.x) lidx[p] = (uint16_t)rank[slot_tmp[p]];
}

// Slices.  A tile's rows are ordered by length and taken 8 at a time; the
// records of a slice are stored step by step, 4 records of each of its 8
// rows per step: record 32 s + 4 r + q of the slice is entry 4 s + q of its
// row r, so the 32 lanes of a warp (4 per row) read one contiguous run.  In
// list order the same loads touched eight separate runs (29 L1 wavefronts a
// warp for a step's FP64 records where 7 suffice), and the two gathers ran at
// 70-83 % of the L1 data pipe.  Rows shorter than their slice are padded with
// zero gradients at their first entry's rank: ordering the 64 rows by length
// first keeps the pads at 5 % of the records (14 % in list order, measured on
// the jittered bar's lists).
//
// Block per tile (R threads or more): the row order and the slices' steps.
__global__ void __launch_bounds__(64) k_slice_rows(int32_t n, int32_t R, const int64_t* __restrict__ ptr,
                                                   uint8_t* __restrict__ ord, int32_t* __restrict__ steps,
                                                   int32_t* __restrict__ most) {
  __shared__ int32_t len[64], sorted[64];
  const int64_t t = blockIdx.x;
  const int i = threadIdx.x;
  const int64_t r = t * R + i;
  if (i < R) len[i] = r < n ? (int32_t)(ptr[r + 1] - ptr[r]) : -1;
  __syncthreads();
  if (i < R) {
    const int mine = len[i];
    int pos = 0;  // rows longer than this one, or as long and before it
    for (int k = 0; k < R; ++k) pos += len[k] > mine || (len[k] == mine && k < i);
    ord[t * R + pos] = (uint8_t)i;
    sorted[pos] = mine;
  }
  __syncthreads();
  if (i < R / 8) steps[t * (R / 8) + i] = (max(sorted[8 * i], 0) + 3) / 4;
  if (i == 0) {
    int sum = 0;
    for (int k = 0; k < R; k += 8) sum += (max(sorted[k], 0) + 3) / 4;
    atomicMax(most, sum);
  }
}

// rbase[row] = the record of the row's first entry (entry k: + 32 (k / 4) + k % 4)
__global__ void k_slice_base(int32_t n, int32_t R, int64_t slots, const uint8_t* __restrict__ ord,
                             const int64_t* __restrict__ sstep, int64_t* __restrict__ rbase) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= slots) return;
  const int64_t row = k / R * R + ord[k];
  if (row < n) rbase[row] = 32 * sstep[k >> 3] + 4 * (k & 7);
}

__device__ __forceinline__ int64_t rec_of(int64_t base, int64_t k) { return base + 32 * (k >> 2) + (k & 3); }

// Four lanes per slot of a tile (so a warp writes a slice step by step): put
// is called for every record of the slot's row, with the list position p of
// its entry, or p < 0 and the row's first position for a pad.
template <typename F>
__device__ __forceinline__ void for_slot_records(int32_t n, int32_t R, int64_t slots, const SliceView& v,
                                                 const int64_t* ptr, F put) {
  const int64_t th = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t slot = th >> 2;
  if (slot >= slots) return;
  const int q = (int)(th & 3);
  const int64_t row = slot / R * R + v.ord[slot];
  const int64_t b = row < n ? ptr[row] : 0, len = row < n ? ptr[row + 1] - b : 0;
  const int64_t s0 = v.sstep[slot >> 3], s1 = v.sstep[(slot >> 3) + 1];
  for (int64_t s = s0; s < s1; ++s) {
    const int64_t k = 4 * (s - s0) + q;
    put(32 * s + 4 * (slot & 7) + q, k < len ? b + k : (int64_t)-1, len > 0 ? b : (int64_t)-1);
  }
}

// records from gradients in list order (pos: where entry p's gradient is)
__global__ void k_pack_f32(int32_t n, int32_t R, int64_t slots, SliceView v, const int64_t* __restrict__ ptr,
                           const uint16_t* __restrict__ lidx, const double* __restrict__ gx,
                           const double* __restrict__ gy, const double* __restrict__ gz,
                           const int64_t* __restrict__ pos, float4* __restrict__ out) {
  for_slot_records(n, R, slots, v, ptr, [&](int64_t rec, int64_t p, int64_t first) {
    float4 o = make_float4(0.f, 0.f, 0.f, __int_as_float(first >= 0 ? (int)lidx[first] : 0));
    if (p >= 0) {
      const int64_t g = pos ? pos[p] : p;
      o = make_float4((float)gx[g], (float)gy[g], (float)gz[g], __int_as_float((int)lidx[p]));
    }
    out[rec] = o;
  });
}

__global__ void k_pack_f64(int32_t n, int32_t R, int64_t slots, SliceView v, const int64_t* __restrict__ ptr,
                           const uint16_t* __restrict__ lidx, const double* __restrict__ gx,
                           const double* __restrict__ gy, const double* __restrict__ gz,
                           const int64_t* __restrict__ pos, void* __restrict__ out) {
  double2* xy = (double2*)out;
  double* z = (double*)(xy + v.nrec);
  uint16_t* l = (uint16_t*)(z + v.nrec);
  for_slot_records(n, R, slots, v, ptr, [&](int64_t rec, int64_t p, int64_t first) {
    const int64_t g = p < 0 ? 0 : (pos ? pos[p] : p);
    xy[rec] = p >= 0 ? make_double2(gx[g], gy[g]) : make_double2(0.0, 0.0);
    z[rec] = p >= 0 ? gz[g] : 0.0;
    l[rec] = p >= 0 ? lidx[p] : (first >= 0 ? lidx[first] : (uint16_t)0);
  });
}

// float column records from the float row records: entry p of the columns is
// entry pos[p] of the rows, in row trow[p]
__global__ void k_pack_t32(int32_t n, int32_t R, int64_t slots, SliceView v, const int64_t* __restrict__ ptr,
                           const uint16_t* __restrict__ lidx, const float4* __restrict__ in,
                           const int32_t* __restrict__ trow, const int64_t* __restrict__ pos,
                           const int64_t* __restrict__ rowptr, const int64_t* __restrict__ rbase,
                           float4* __restrict__ out) {
  for_slot_records(n, R, slots, v, ptr, [&](int64_t rec, int64_t p, int64_t first) {
    float4 o = make_float4(0.f, 0.f, 0.f, __int_as_float(first >= 0 ? (int)lidx[first] : 0));
    if (p >= 0) {
      const int32_t r = trow[p];
      const float4 x = in[rec_of(rbase[r], pos[p] - rowptr[r])];
      o = make_float4(x.x, x.y, x.z, __int_as_float((int)lidx[p]));
    }
    out[rec] = o;
  });
}

// the pads alone (the shape kernel wrote the real records)
__global__ void k_pad_f32(int32_t n, int32_t R, int64_t slots, SliceView v, const int64_t* __restrict__ ptr,
                          const uint16_t* __restrict__ lidx, float4* __restrict__ out) {
  for_slot_records(n, R, slots, v, ptr, [&](int64_t rec, int64_t p, int64_t first) {
    if (p < 0) out[rec] = make_float4(0.f, 0.f, 0.f, __int_as_float(first >= 0 ? (int)lidx[first] : 0));
  });
}

// Entry order for conflict-free reads of the staged neighbour data.  In the
// gathers the KG lanes of a row (column) take its entries KG at a time, and
// the lanes of a warp read the staged 16-byte vectors of their current
// entries in one instruction, 8 lanes at a time: lanes of such a group whose
// tile ranks l differ but agree modulo NC = 8 (the vectors' bank period) are
// served one after another, lanes with the same l by one broadcast.  This
// reorders the entries within each row so that, at every step, the lanes of
// each group of GL = 8 lanes hold, per class l mod NC, one rank only wherever
// the row's remaining entries allow (greedy, lanes in order, each taking its
// first entry whose class is free or holds the same rank); a row keeps all
// its entries, only their order changes.
// pos (the identity on entry) is permuted with lidx.  One warp per warp of the gather's
// blocks, four warps per block.
constexpr int kBankCap = 2048;  // entries of one warp's rows that its pass stages in shared memory

template <int KG, int NC, int GL>
__global__ void __launch_bounds__(128) k_bank_order(int32_t n, int32_t R, int64_t nwarps,
                                                    const uint8_t* __restrict__ ord,
                                                    const int64_t* __restrict__ ptr, uint16_t* lidx, int64_t* pos) {
  __shared__ int held_s[4][32];
  __shared__ uint16_t sl_s[4][kBankCap], so_s[4][kBankCap];  // ranks, and offsets in the row before
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (w >= nwarps) return;  // whole warps leave together
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  int* held = held_s[wi] + (lane / GL) * NC;  // this lane's group: the rank held per class
  const int wpt = R * KG / 32;  // warps per tile
  const int64_t c = (w / wpt) * R + ord[(w / wpt) * R + (w % wpt) * (32 / KG) + lane / KG];
  const int q = lane & (KG - 1);
  int64_t b = 0, e = 0;
  if (c < n) { b = ptr[c]; e = ptr[c + 1]; }
  const int len = (int)(e - b);
  // the warp's rows one after another in shared memory, where they fit
  int x = q == 0 ? len : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  const int total = __shfl_sync(0xffffffffu, x, 31);
  const int off = __shfl_sync(0xffffffffu, x - (q == 0 ? len : 0), lane & ~(KG - 1));
  const bool fast = total <= kBankCap;  // warp-uniform
  uint16_t* sl = sl_s[wi] + off;
  uint16_t* so = so_s[wi] + off;
  if (fast)
    for (int k = q; k < len; k += KG) { sl[k] = lidx[b + k]; so[k] = (uint16_t)k; }
  __syncwarp();
  int steps = (len + KG - 1) / KG;
#pragma unroll
  for (int o = 16; o; o >>= 1) steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, o));
  for (int s = 0; s < steps; ++s) {
    const int slot = s * KG + q;
    held_s[wi][lane] = -1;
    __syncwarp();
    for (int turn = 0; turn < 32; ++turn) {
      if (lane == turn && slot < len) {
        if (fast) {
          int pick = slot;
          for (int k = slot; k < len; ++k) {
            const int l = sl[k], h = held[l & (NC - 1)];
            if (h < 0 || h == l) { pick = k; break; }
          }
          if (pick != slot) {
            const uint16_t t1 = sl[pick]; sl[pick] = sl[slot]; sl[slot] = t1;
            const uint16_t t2 = so[pick]; so[pick] = so[slot]; so[slot] = t2;
          }
          const int l = sl[slot];
          if (held[l & (NC - 1)] < 0) held[l & (NC - 1)] = l;
        } else {  // rows too long for shared memory: the same pass in place
          int64_t pick = b + slot;
          for (int64_t k = b + slot; k < e; ++k) {
            const int l = lidx[k], h = held[l & (NC - 1)];
            if (h < 0 || h == l) { pick = k; break; }
          }
          if (pick != b + slot) {
            const uint16_t t1 = lidx[pick]; lidx[pick] = lidx[b + slot]; lidx[b + slot] = t1;
            const int64_t t2 = pos[pick]; pos[pick] = pos[b + slot]; pos[b + slot] = t2;
          }
          const int l = lidx[b + slot];
          if (held[l & (NC - 1)] < 0) held[l & (NC - 1)] = l;
        }
      }
      __syncwarp();
    }
  }
  if (fast)
    for (int k = q; k < len; k += KG) {
      lidx[b + k] = sl[k];
      pos[b + k] = b + so[k];
    }
}

// the records of each row in a new order: entry p takes the record of entry
// pos[p] of the same row (pads stay)
__global__ void k_gather_rec32(int32_t n, int32_t R, int64_t slots, SliceView v, const int64_t* __restrict__ ptr,
                               const int64_t* __restrict__ pos, const float4* __restrict__ in,
                               float4* __restrict__ out) {
  for_slot_records(n, R, slots, v, ptr, [&](int64_t rec, int64_t p, int64_t first) {
    int64_t from = rec;
    if (p >= 0) {
      const int64_t k = p - first;
      from = rec_of(rec - 32 * (k >> 2) - (k & 3), pos[p] - first);
    }
    out[rec] = in[from];
  });
}

// the same for the planes of FP64 records
__global__ void k_gather_rec64(int32_t n, int32_t R, int64_t slots, SliceView v, const int64_t* __restrict__ ptr,
                               const int64_t* __restrict__ pos, const void* __restrict__ in, void* __restrict__ out) {
  const double2* xy = (const double2*)in;
  const double* z = (const double*)(xy + v.nrec);
  const uint16_t* l = (const uint16_t*)(z + v.nrec);
  double2* oxy = (double2*)out;
  double* oz = (double*)(oxy + v.nrec);
  uint16_t* ol = (uint16_t*)(oz + v.nrec);
  for_slot_records(n, R, slots, v, ptr, [&](int64_t rec, int64_t p, int64_t first) {
    int64_t from = rec;
    if (p >= 0) {
      const int64_t k = p - first;
      from = rec_of(rec - 32 * (k >> 2) - (k & 3), pos[p] - first);
    }
    oxy[rec] = xy[from];
    oz[rec] = z[from];
    ol[rec] = l[from];
  });
}

// NSNI's second derivatives in the records' layout (planes of nrec values)
template <bool F64>
__device__ __forceinline__ void put_second(void* out, int64_t nrec, int64_t rec, const double v[6]) {
  if constexpr (F64) {
    double2* o = (double2*)out;
#pragma unroll
    for (int c = 0; c < 3; ++c) o[c * nrec + rec] = make_double2(v[2 * c], v[2 * c + 1]);
  } else {
    ((float4*)out)[rec] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
    ((float2*)((float4*)out + nrec))[rec] = make_float2((float)v[4], (float)v[5]);
  }
}

template <bool F64>
__global__ void k_pack_second(int32_t n, int32_t R, int64_t slots, SliceView v, const int64_t* __restrict__ ptr,
                              const int64_t* __restrict__ pos, NsniS src, void* __restrict__ out) {
  for_slot_records(n, R, slots, v, ptr, [&](int64_t rec, int64_t p, int64_t) {
    double x[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (p >= 0) {
      const int64_t g = pos ? pos[p] : p;
#pragma unroll
      for (int c = 0; c < 6; ++c) x[c] = src.v[c][g];
    }
    put_second<F64>(out, v.nrec, rec, x);
  });
}

template <bool F64>
__global__ void k_gather_second(int32_t n, int32_t R, int64_t slots, SliceView v, const int64_t* __restrict__ ptr,
                                const int64_t* __restrict__ pos, const void* __restrict__ in,
                                void* __restrict__ out) {
  for_slot_records(n, R, slots, v, ptr, [&](int64_t rec, int64_t p, int64_t first) {
    int64_t from = rec;
    if (p >= 0) {
      const int64_t k = p - first;
      from = rec_of(rec - 32 * (k >> 2) - (k & 3), pos[p] - first);
    }
    if constexpr (F64) {
#pragma unroll
      for (int c = 0; c < 3; ++c) ((double2*)out)[c * v.nrec + rec] = ((const double2*)in)[c * v.nrec + from];
    } else {
      ((float4*)out)[rec] = ((const float4*)in)[from];
      ((float2*)((float4*)out + v.nrec))[rec] = ((const float2*)((const float4*)in + v.nrec))[from];
    }
  });
}

__global__ void k_iota64(int64_t m, int64_t* __restrict__ out) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e < m) out[e] = e;
}

// One record as a lane holds it: the gradient in the arithmetic's type and
// the tile rank.  FP64 records are three planes (x and y, z, rank) of nrec
// values each, so each load of a warp is contiguous.
template <bool F64>
struct Rec;
template <>
struct Rec<false> {
  float4 v;
  __device__ __forceinline__ float x() const { return v.x; }
  __device__ __forceinline__ float y() const { return v.y; }
  __device__ __forceinline__ float z() const { return v.z; }
  __device__ __forceinline__ int l() const { return __float_as_int(v.w); }
};
template <>
struct Rec<true> {
  double2 a;
  double b;
  uint16_t r;
  __device__ __forceinline__ double x() const { return a.x; }
  __device__ __forceinline__ double y() const { return a.y; }
  __device__ __forceinline__ double z() const { return b; }
  __device__ __forceinline__ int l() const { return (int)r; }
};
__device__ __forceinline__ void load_rec(const void* pk, int64_t, int64_t rec, Rec<false>& o) {
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o.v.x), "=f"(o.v.y), "=f"(o.v.z), "=f"(o.v.w) : "l"((const float4*)pk + rec));
}
__device__ __forceinline__ void load_rec(const void* pk, int64_t nrec, int64_t rec, Rec<true>& o) {
  const double2* xy = (const double2*)pk;
  const double* z = (const double*)(xy + nrec);
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(o.a.x), "=d"(o.a.y) : "l"(xy + rec));
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(o.b) : "l"(z + rec));
  asm("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(o.r) : "l"((const uint16_t*)(z + nrec) + rec));
}

// N values per rank staged in shared memory: 16-byte vectors (4 floats or 2
// doubles) of all ranks one after another, then the values left over as
// arrays, ld ranks each.  A lane's read of 9 values is 3 (float) or 5
// (double) instructions.  Lanes with distinct ranks modulo 8 among 8
// neighbouring lanes read distinct banks; a warp's random ranks cost a 16-byte
// read 8.3 wavefronts where four 4-byte reads cost 11.0 and two 8-byte reads
// 10.3 (counted on the jittered bar's lists).  ld is a multiple of 4, so what
// follows the values is aligned too.
__host__ __device__ constexpr int staged_ld(int cnt) { return (cnt + 3) & ~3; }
template <typename V, int N>
struct Staged {
  static constexpr int W = 16 / (int)sizeof(V), NV = N / W;
  V* base;
  int ld;
  __device__ __forceinline__ V* end() const { return base + N * ld; }
  // value k of rank l
  __device__ __forceinline__ V& at(int l, int k) const {
    return k < W * NV ? base[W * ((k / W) * ld + l) + k % W] : base[k * ld + l];
  }
  // vector k of rank l
  __device__ __forceinline__ void put(int l, int k, const float4& x) const {
    reinterpret_cast<float4*>(base)[k * ld + l] = x;
  }
  __device__ __forceinline__ void put(int l, int k, const double2& x) const {
    reinterpret_cast<double2*>(base)[k * ld + l] = x;
  }
  __device__ __forceinline__ void load(int l, V* v) const {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if constexpr (W == 4) {
        const float4 x = reinterpret_cast<const float4*>(base)[k * ld + l];
        v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
      } else {
        const double2 x = reinterpret_cast<const double2*>(base)[k * ld + l];
        v[2 * k] = x.x; v[2 * k + 1] = x.y;
      }
    }
#pragma unroll
    for (int k = W * NV; k < N; ++k) v[k] = base[k * ld + l];
  }
};

// 32 bytes at a 32-byte boundary
__device__ __forceinline__ void load_sector(const double* p, double v[4]) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// A lane's way through its row's records: KG lanes per row (4, 8 or 16), the
// lane's entries KG apart in list order, which is a stride of KG / 4 steps.
// ns is uniform over a slice's lanes when KG = 4.
template <int KG>
struct RowWalk {
  int64_t rec;  // the lane's first record
  int nit;      // its records (pads among them)
  __device__ __forceinline__ RowWalk(const SliceView& v, int64_t slot0, int slot, int lane) {
    const int64_t sl = (slot0 + slot) >> 3;
    const int64_t s0 = v.sstep[sl];
    const int ns = (int)(v.sstep[sl + 1] - s0), h = lane >> 2;
    rec = 32 * (s0 + h) + 4 * (slot & 7) + (lane & 3);
    nit = (ns - h + KG / 4 - 1) / (KG / 4);
  }
  __device__ __forceinline__ int64_t at(int k) const { return rec + (int64_t)(8 * KG) * k; }
};

// The records of a slice past its rows' first KU steps, on their way to L2 while
// the tile's neighbours are staged (each plane 64-byte aligned: whole steps).
template <bool F64, int KG>
__device__ __forceinline__ void prefetch_rest(const void* pk, const SliceView& v, int64_t slot0, int slot, int ku) {
  if ((threadIdx.x & (8 * KG - 1)) != 0) return;
  const int64_t sl = (slot0 + slot) >> 3;
  const int64_t s0 = v.sstep[sl] + ku * (KG / 4), n = 32 * (v.sstep[sl + 1] - s0), r = 32 * s0;
  if (n <= 0) return;
  const char* b = (const char*)pk;
  const auto fetch = [](const char* p, int64_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"((unsigned)bytes) : "memory");
  };
  fetch(b + 16 * r, 16 * n);
  if (F64) {
    fetch(b + 16 * v.nrec + 8 * r, 8 * n);
    fetch(b + 24 * v.nrec + 2 * r, 2 * n);
  }
}

// The six S values of one NSNI record.
template <bool F64>
struct SRec;
template <>
struct SRec<false> {
  float4 a;
  float2 b;
  __device__ __forceinline__ void load(const void* base, int64_t nrec, int64_t rec) {
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w)
        : "l"((const float4*)base + rec));
    asm("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];"
        : "=f"(b.x), "=f"(b.y)
        : "l"((const float2*)((const float4*)base + nrec) + rec));
  }
  template <typename A>
  __device__ __forceinline__ void get(A s[6]) const {
    s[0] = (A)a.x; s[1] = (A)a.y; s[2] = (A)a.z; s[3] = (A)a.w; s[4] = (A)b.x; s[5] = (A)b.y;
  }
};
template <>
struct SRec<true> {
  double2 a[3];
  __device__ __forceinline__ void load(const void* base, int64_t nrec, int64_t rec) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];"
          : "=d"(a[c].x), "=d"(a[c].y)
          : "l"((const double2*)base + c * nrec + rec));
  }
  template <typename A>
  __device__ __forceinline__ void get(A s[6]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) { s[2 * c] = (A)a[c].x; s[2 * c + 1] = (A)a[c].y; }
  }
};

// the staged displacement values of a rank: three doubles, or three floats and a pad
template <bool F64>
struct DispStage {
  using V = float;
  static constexpr int N = 4;
};
template <>
struct DispStage<true> {
  using V = double;
  static constexpr int N = 3;
};

template <bool F64>
using StagedDisp = Staged<typename DispStage<F64>::V, DispStage<F64>::N>;

// The ranks a thread stages, in its order: the first ones are read before the
// wait for the kernel before (the sets' rows have room for jmax ids, so a rank
// past the tile's count reads stale ids that are not used).
template <int KG>
struct StageIds {
  static constexpr int K = 16 / KG;
  int32_t id[K];
  const int32_t* js;
  __device__ __forceinline__ StageIds(const int32_t* js_, int32_t jmax) : js(js_) {
#pragma unroll
    for (int u = 0; u < K; ++u) {
      const int l = threadIdx.x + u * blockDim.x;
      id[u] = l < jmax ? js[l] : 0;
    }
  }
  // f(rank, node) for this thread's ranks below cnt
  template <typename F>
  __device__ __forceinline__ void each(int cnt, F f) const {
#pragma unroll
    for (int u = 0; u < K; ++u) {
      const int l = threadIdx.x + u * blockDim.x;
      if (l < cnt) f(l, (int64_t)id[u]);
    }
    for (int l = threadIdx.x + K * blockDim.x; l < cnt; l += blockDim.x) f(l, (int64_t)js[l]);
  }
};

// a thread per staged node
template <bool F64, int KG>
__device__ __forceinline__ void stage_disp(const StageIds<KG>& ids, int cnt, const double* v, const double* ref,
                                           const StagedDisp<F64>& out) {
  ids.each(cnt, [&](int l, int64_t j) {
    const double x0 = v[3 * j], x1 = v[3 * j + 1], x2 = v[3 * j + 2];
    if constexpr (F64) {
      out.put(l, 0, make_double2(x0, x1));
      out.at(l, 2) = x2;
    } else {
      out.put(l, 0, make_float4((float)(x0 - ref[0]), (float)(x1 - ref[1]), (float)(x2 - ref[2]), 0.f));
    }
  });
}

// The sums of a step, cleared by the first 32 threads of a block: a tile of 8
// rows has no more (a loop over the slots cost the joined kernels spills).
template <typename T>
__device__ __forceinline__ void clear_slots(T* v) {
  static_assert(kSlots == 64, "two a thread");
  v[threadIdx.x] = T(0);
  v[threadIdx.x + 32] = T(0);
}
__device__ __forceinline__ void clear_counts(StepAccum* acc) {
  clear_slots(acc->newton_iters);
  clear_slots(acc->plastic);
}

// FULL: F - I is formed besides G0.  Without it the gather stages and reads
// the increments alone, half the shared-memory traffic and sums: at 130 k nodes
// FP64 ran at 75 % of the L1 data pipe with both, half of it staged reads.
// NS: the NSNI gradients of the incremental displacement gradient ride
// along, H_i(k, q) = sum_J S_q(i, J) du_J,k, in mixed precision formed like L
// as sum_J S_q (du_J - du_i) + du_i,k sum_J S_q (FINT.F90:728-737 layout).
template <bool F64, int KG, bool NS, bool FULL>
constexpr int defgrad_blocks() {  // blocks per SM the register cap asks for
  const int w = NS ? 8 : (F64 && FULL ? 12 : 16);
  return w / KG > 0 ? w / KG : 1;
}

struct NoStress {};
template <typename SA>
constexpr bool kHasStress = !std::is_same<SA, NoStress>::value;

// SA: StressArgs where the block goes on to the stress update of its rows,
// NoStress else.  What bounds a step of a few thousand nodes is the latency of
// its kernels, one after the other: with the rows' G0 at hand behind a block
// barrier, the update needs no launch of its own.  It takes 128 registers, so
// two blocks of 256 threads an SM; defgrad_stress_fits has the rule.
template <typename A, bool F64, bool INTERP, int KG, int KU, bool NS, bool FULL, typename SA = NoStress>
__global__ void __launch_bounds__(kHasStress<SA> && KG == 16 ? 512 : 64 * KG,
                                  kHasStress<SA> ? (KG == 4 ? 2 : 1) : defgrad_blocks<F64, KG, NS, FULL>())
    k_defgrad_t(int32_t n, int32_t R, int32_t jmax, NsniTiles ns, SliceView sv, const int64_t* __restrict__ rowptr,
                const void* __restrict__ pk, const int32_t* __restrict__ jset, const int32_t* __restrict__ jcnt,
                const double* dsp, const double* dsp_tot, const double* __restrict__ sdphi,
                const double* __restrict__ shp, double* dsp_tot_phy, double* fg, StepAccum* acc, SA sa) {
  extern __shared__ __align__(16) double sm[];
  const int64_t t = blockIdx.x;
  const int cnt = jcnt[t];
  const StageIds<KG> ids(jset + t * (int64_t)jmax, jmax);
  // Staged neighbour displacements, du_J (FULL: and u_J).  FP64 as doubles;
  // mixed as float offsets from the tile's first node r0 (du_J - du_r0,
  // u_J - u_r0; one 16-byte vector with a pad), half the shared-memory
  // traffic: the differences d_J - d_i are formed between offsets, exact up
  // to float rounding of the offsets.
  using SV = typename DispStage<F64>::V;
  constexpr int SN = DispStage<F64>::N;
  const Staged<SV, SN> sd{reinterpret_cast<SV*>(sm), staged_ld(cnt)};
  const Staged<SV, SN> su{sd.end(), sd.ld};
  const int64_t r0 = t * R;
  const int slot = threadIdx.x / KG;
  const int64_t i = r0 + sv.ord[r0 + slot];
  const int q = threadIdx.x & (KG - 1);
  const unsigned gmask = group_mask<KG>();
  const bool valid = i < n;
  // this lane's first KU packed records are requested before the staging,
  // so their latency overlaps it
  if (!NS && (!F64 || kHasStress<SA>) && sv.ahead) prefetch_rest<F64, KG>(pk, sv, r0, slot, KU);
  const RowWalk<KG> walk(sv, r0, slot, q);
  const int nit = valid ? walk.nit : 0;
  constexpr bool kPipe = !NS && (!F64 || KU <= 2);
  int64_t p0 = 0, pend = 0;  // list positions, for the shape values
  if (INTERP && valid) {
    p0 = rowptr[i] + q;
    pend = rowptr[i + 1];
  }
  Rec<F64> cur[KU];
  SRec<F64> csr[NS ? KU : 1];
  bool have = nit >= KU;
  if (have) {
#pragma unroll
    for (int u = 0; u < KU; ++u) {
      load_rec(pk, sv.nrec, walk.at(u), cur[u]);
      if constexpr (NS) csr[u].load(ns.srow, sv.nrec, walk.at(u));
    }
  }
  grid_wait();
  if (acc && blockIdx.x == 0 && threadIdx.x < 32) {
    // (no counts of this step alone where it joins: a call's last step is not one of these)
    if constexpr (kHasStress<SA>) clear_slots(acc->ke);
    else clear_counts(acc);
  }
  double ur[3] = {0.0, 0.0, 0.0}, dr[3] = {0.0, 0.0, 0.0};
  if (!F64) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dr[k] = dsp[3 * r0 + k];
      if (FULL) ur[k] = dsp_tot[3 * r0 + k];
    }
  }
  stage_disp<F64, KG>(ids, cnt, dsp, dr, sd);
  if (FULL) stage_disp<F64, KG>(ids, cnt, dsp_tot, ur, su);
  __syncthreads();
  if (valid) {
    double ui[3] = {0.0, 0.0, 0.0}, di[3];
    A fu[3], fd[3];  // this row's values as the staged ones are held
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      di[k] = dsp[3 * i + k];
      fd[k] = F64 ? (A)di[k] : (A)(float)(di[k] - dr[k]);
      if (FULL) {
        ui[k] = dsp_tot[3 * i + k];
        fu[k] = F64 ? (A)ui[k] : (A)(float)(ui[k] - ur[k]);
      }
    }
    A F[FULL ? 9 : 1], L[9];
    double H[NS ? 18 : 1];  // NSNI: exact products of the float S and differences, summed in double
#pragma unroll
    for (int k = 0; k < 9; ++k) L[k] = A(0);
#pragma unroll
    for (int k = 0; k < (FULL ? 9 : 1); ++k) F[k] = A(0);
#pragma unroll
    for (int k = 0; k < (NS ? 18 : 1); ++k) H[k] = 0.0;
    double ph[3] = {0.0, 0.0, 0.0};
    // One entry: F += (u_J - u_i) (x) g, L += (d_J - d_i) (x) g (+ phi d_J),
    // H(k, q) += S_q (d_J - d_i)_k.
    auto body = [&](int it, const Rec<F64>& rec, const SRec<F64>& sr) {
      const A g[3] = {(A)rec.x(), (A)rec.y(), (A)rec.z()};
      const int l = rec.l();
      SV v[SN];
      A d[3];
      sd.load(l, v);
#pragma unroll
      for (int k = 0; k < 3; ++k) d[k] = (A)v[k] - fd[k];
      if constexpr (FULL) {
        SV w[SN];
        su.load(l, w);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const A u = (A)w[k] - fu[k];
          F[3 * k] += u * g[0]; F[3 * k + 1] += u * g[1]; F[3 * k + 2] += u * g[2];
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        L[3 * k] += d[k] * g[0]; L[3 * k + 1] += d[k] * g[1]; L[3 * k + 2] += d[k] * g[2];
      }
      if constexpr (NS) {
        double sq[6];
        sr.get(sq);
        // FP64: du_J itself
        const double e0 = F64 ? (double)v[0] : (double)d[0], e1 = F64 ? (double)v[1] : (double)d[1],
                     e2 = F64 ? (double)v[2] : (double)d[2];
#pragma unroll
        for (int c = 0; c < 6; ++c) { H[c] += sq[c] * e0; H[6 + c] += sq[c] * e1; H[12 + c] += sq[c] * e2; }
      }
      if (INTERP) {
        const int64_t p = p0 + (int64_t)KG * it;
        if (p < pend) {  // (not a pad)
          const double s = shp[p];
#pragma unroll
          for (int k = 0; k < 3; ++k) ph[k] += s * (F64 ? (double)v[k] : dr[k] + (double)v[k]);
        }
      }
    };
    // Each lane sums its entries in list order.  Where the registers allow
    // (kPipe) the next KU records are requested before this KU's sums, so a
    // lane keeps loads in flight while it computes.
    int it = 0;
    while (have) {
      const bool hn = it + 2 * KU <= nit;
      Rec<F64> nxt[KU];
      if constexpr (kPipe) {
#pragma unroll
        for (int u = 0; u < KU; ++u) {
          if (hn) load_rec(pk, sv.nrec, walk.at(it + KU + u), nxt[u]);
          else nxt[u] = cur[u];
        }
      }
#pragma unroll
      for (int u = 0; u < KU; ++u) body(it + u, cur[u], csr[NS ? u : 0]);
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        if constexpr (kPipe) {
          cur[u] = nxt[u];
        } else if (hn) {
          load_rec(pk, sv.nrec, walk.at(it + KU + u), cur[u]);
          if constexpr (NS) csr[u].load(ns.srow, sv.nrec, walk.at(it + KU + u));
        }
      }
      it += KU;
      have = hn;
    }
    for (; it < nit; ++it) {
      Rec<F64> rec;
      load_rec(pk, sv.nrec, walk.at(it), rec);
      SRec<F64> sr;
      if constexpr (NS) sr.load(ns.srow, sv.nrec, walk.at(it));
      body(it, rec, sr);
    }
#pragma unroll
    for (int o = 1; o < KG; o <<= 1) {
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        if constexpr (FULL) F[k] += __shfl_xor_sync(gmask, F[k], o);
        L[k] += __shfl_xor_sync(gmask, L[k], o);
      }
      if constexpr (NS) {
#pragma unroll
        for (int k = 0; k < 18; ++k) H[k] += __shfl_xor_sync(gmask, H[k], o);
      }
      if (INTERP) {
#pragma unroll
        for (int k = 0; k < 3; ++k) ph[k] += __shfl_xor_sync(gmask, ph[k], o);
      }
    }
    if (q == 0) {
      if constexpr (NS) {
        double ss[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (!F64)
#pragma unroll
          for (int c = 0; c < 6; ++c) ss[c] = ns.ssum[6 * i + c];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int c = 0; c < 6; ++c)
            ns.hq[(6 * k + c) * fg_ld(n) + i] = F64 ? H[6 * k + c] : H[6 * k + c] + di[k] * ss[c];
      }
      const double sd3[3] = {sdphi[3 * i], sdphi[3 * i + 1], sdphi[3 * i + 2]};
      const int64_t ld = fg_ld(n);
      double h[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) h[k] = (double)L[k] + di[k / 3] * sd3[k % 3];
      store_g0(fg, ld, i, !F64, h);
      if constexpr (FULL) {
#pragma unroll
        for (int k = 0; k < 9; ++k) h[k] = (double)F[k] + ui[k / 3] * sd3[k % 3];
        store_fmi(fg, ld, i, h);
      }
      if (INTERP) {
#pragma unroll
        for (int k = 0; k < 3; ++k) dsp_tot_phy[3 * i + k] += ph[k];
      }
    }
  }
  if constexpr (kHasStress<SA>) {
    __shared__ double smd[32];
    __shared__ unsigned long long smu[32];
    __syncthreads();  // G0 of the tile's rows, written by other threads of this block
    double work = 0.0;
    unsigned long long iters = 0, npl = 0;
    unsigned st = 0;
    const int64_t row = r0 + threadIdx.x;
    if ((int)threadIdx.x < R && row < n) {
      Trial<A, true> w;
      stress_trial<A, true, false, true>(sa, row, w);
      stress_finish<A, A, true, false, true>(sa, row, w, -1.0, work, iters, npl, st);
    }
    stress_reduce<A, false>(sa, work, iters, npl, st, smd, smu);
  }
}

// One DOF m = 3 J + q after its column sum fi (and body-force sum fe):
// fixity, acceleration and corrector (MAIN.F90:432-488), the energy and
// reaction sums, and the next step's predictor (MAIN.F90:353-355).
__device__ __forceinline__ void correct_dof(const TiledForceArgs& a, int64_t J, int q, double fi, double fe,
                                            double& ke, double& ee, double& pr, int& body, unsigned& st) {
  const int64_t m = 3 * J + q;
  const double dt = a.ndt ? a.ndt[J] : a.dt;
  if (!isfinite(fi)) st |= MEGA_ST_NONFINITE;
  const double mass = a.mass[m];
  const double fe_old = a.fext[m], d_old = a.dsp[m];
  // read with the rest: behind the stores below it would cost another trip to memory
  const double u_old = a.predict ? a.dsp_tot[m] : 0.0;
  double v = a.vel[m], acc;
  const int code = a.ebc[m];
  body = a.body_id ? a.body_id[J] : 1;
  const double damp = a.mats[a.matidx[J]].damp;
  if (code == 1 || code == 2) {  // MAIN.F90:438-445 (fixed), 447-470 (prescribed velocity)
    v = code == 1 ? 0.0 : a.vel2[q];
    acc = 0.0;
    pr = -fi;
    fe = -fi;
  } else {  // MAIN.F90:472-481
    const double mpdc = damp * mass;
    acc = (fe - fi - mpdc * v) / (mass + 0.5 * dt * mpdc);
    v = v + 0.5 * dt * acc;
    pr = 0.0;
  }
  ee = 0.5 * (fe + fe_old) * d_old;
  ke = 0.5 * mass * v * v;
  a.fext[m] = fe;
  if (!a.predict) {
    a.fint[m] = fi;
    a.acl[m] = acc;
    a.prforce[m] = pr;
  }
  if (a.predict) {  // MAIN.F90:353-355 of the next step
    const double d = dt * v + dt * dt * 0.5 * acc;
    a.dsp[m] = d;
    a.dsp_tot[m] = u_old + d;
    v = v + dt * 0.5 * acc;
  }
  a.vel[m] = v;
}

// The tile's columns after their sums: thread m takes DOF m of the tile
// (component m % 3 of local column m / 3), so every array is read and written
// in contiguous runs (the warps' own columns are in the slices' order, 8
// scattered columns each), then one block reduction of the step sums and one
// atomic per sum into this block's slot.  Reaction sums are formed only by
// warps that hold a fixed DOF.  Every thread of the block takes part.
struct ColumnSums {
  double f[3 * 64];  // force, and body force, of DOF m
  double e[3 * 64];
  double red[6 * 8];
};

// the lines finish_columns will read, asked for while the sums are formed
__device__ __forceinline__ void prefetch_columns(const TiledForceArgs& a, int64_t c0) {
  const int64_t m = 3 * c0 + threadIdx.x;
  if (threadIdx.x >= 3 * a.R || (threadIdx.x & 3) || m >= 3 * (int64_t)a.n) return;
  prefetch_l2(a.mass + m);
  prefetch_l2(a.fext + m);
  prefetch_l2(a.vel + m);
  prefetch_l2(a.dsp + m);
  prefetch_l2(a.dsp_tot + m);
}

template <bool BODY>
__device__ __forceinline__ void finish_columns(const TiledForceArgs& a, int64_t c0, ColumnSums& cs, unsigned st) {
  __syncthreads();
  const int tid = threadIdx.x, ndof = 3 * a.R, nw = (ndof + 31) >> 5, wid = tid >> 5;
  if (wid < nw) {  // whole warps
    double ke = 0.0, ee = 0.0, pr = 0.0;
    int body = 0;
    const int q = tid % 3;
    const int64_t J = c0 + tid / 3;
    if (tid < ndof && J < a.n) correct_dof(a, J, q, cs.f[tid], BODY ? cs.e[tid] : 0.0, ke, ee, pr, body, st);
    double v[8] = {ke, ee, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      v[1] += __shfl_xor_sync(0xffffffffu, v[1], o);
    }
    if (__any_sync(0xffffffffu, pr != 0.0)) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        v[2 + k] = (q == k % 3 && body == 1 + k / 3) ? pr : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[2 + k] += __shfl_xor_sync(0xffffffffu, v[2 + k], o);
      }
    }
    if ((tid & 31) == 0)
#pragma unroll
      for (int k = 0; k < 8; ++k) cs.red[wid * 8 + k] = v[k];
  }
  __syncthreads();
  if (tid < 8) {
    double tsum = 0.0;
    for (int w = 0; w < nw; ++w) tsum += cs.red[w * 8 + tid];
    const int sl = blockIdx.x % kSlots;
    double* dst = tid == 0 ? &a.acc->ke[sl] : (tid == 1 ? &a.acc->ee[sl] : &a.acc->tf[tid - 2][sl]);
    if (tsum != 0.0) atomicAdd(dst, tsum);
  }
  if (st) atomicOr(a.status, st);
}

// The staged values of a column tile: T_i (9), NS: with W_i (18), and the body
// force vectors (3, as arrays).  Mixed NS: 27 values and a pad in 7 vectors,
// T_i's first two, then T_i's last beside W_i's last two, then W_i's first
// 16.  FP64 NS: T_i then W_i, 27 values, 216 bytes a rank, so that 1,024 ranks
// fit; its body force is read through the node ids, which are staged instead.
template <typename TS, bool NS>
struct StagedT {
  static constexpr int N = NS ? (sizeof(TS) == 4 ? 28 : 27) : 9;
  static constexpr bool kIds = NS && sizeof(TS) == 8;
  Staged<TS, N> t;
  TS* body;
  int ld;
  static size_t bytes(int maxcnt, bool has_body) {
    return (size_t)staged_ld(maxcnt) * (N * sizeof(TS) + (has_body ? (kIds ? 4 : 3 * sizeof(TS)) : 0));
  }
  __device__ __forceinline__ StagedT(void* base, int cnt)
      : t{reinterpret_cast<TS*>(base), staged_ld(cnt)}, body(t.end()), ld(t.ld) {}
  // the body force vector of rank l
  __device__ __forceinline__ void body_of(const TiledForceArgs& a, int l, double b[3]) const {
    if constexpr (kIds) {
      const double* p = reinterpret_cast<const double*>(a.tmat) + 12 * (int64_t)reinterpret_cast<const int32_t*>(body)[l];
      b[0] = p[9]; b[1] = p[10]; b[2] = p[11];
    } else {
      b[0] = (double)body[l]; b[1] = (double)body[ld + l]; b[2] = (double)body[2 * ld + l];
    }
  }
  // W_l(k, q) at 6 k + q
  __device__ __forceinline__ static TS weight(const TS* v, int j) {
    return sizeof(TS) == 8 ? v[9 + j] : (j < 16 ? v[12 + j] : v[j - 7]);
  }
  template <bool BODY, int KG>
  __device__ __forceinline__ void fill(const TiledForceArgs& a, const StageIds<KG>& ids, int cnt) const {
    ids.each(cnt, [&](int l, int64_t j) {
      if constexpr (sizeof(TS) == 4) {
        const float4* p = reinterpret_cast<const float4*>(a.tmat) + 3 * j;
        const float4 x = p[0], y = p[1], z = p[2];
        t.put(l, 0, x);
        t.put(l, 1, y);
        t.at(l, 8) = z.x;
        if (BODY) { body[l] = z.y; body[ld + l] = z.z; body[2 * ld + l] = z.w; }
        if constexpr (NS) {
          const float4* w = reinterpret_cast<const float4*>(a.ns_w) + 5 * j;
          const float4 w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
          t.put(l, 3, w0);
          t.put(l, 4, w1);
          t.put(l, 5, w2);
          t.put(l, 6, w3);
          t.at(l, 9) = w4.x;
          t.at(l, 10) = w4.y;
        }
      } else {
        const double* p = reinterpret_cast<const double*>(a.tmat) + 12 * j;
        double x[4], y[4], z[4];
        load_sector(p, x);
        load_sector(p + 4, y);
        load_sector(p + 8, z);
        t.put(l, 0, make_double2(x[0], x[1]));
        t.put(l, 1, make_double2(x[2], x[3]));
        t.put(l, 2, make_double2(y[0], y[1]));
        t.put(l, 3, make_double2(y[2], y[3]));
        if constexpr (NS) {
          const double* w = reinterpret_cast<const double*>(a.ns_w) + 20 * j;
          double u[20];
#pragma unroll
          for (int k = 0; k < 5; ++k) load_sector(w + 4 * k, u + 4 * k);
          t.put(l, 4, make_double2(z[0], u[0]));
#pragma unroll
          for (int k = 0; k < 8; ++k) t.put(l, 5 + k, make_double2(u[2 * k + 1], u[2 * k + 2]));
          t.at(l, 26) = u[17];
          if (BODY) reinterpret_cast<int32_t*>(body)[l] = (int32_t)j;
        } else {
          t.at(l, 8) = z[0];
          if (BODY) { body[l] = z[1]; body[ld + l] = z[2]; body[2 * ld + l] = z[3]; }
        }
      }
    });
  }
};

template <bool F64, int KG, int KU, bool NS>
constexpr int force_blocks() {  // blocks per SM the register cap asks for (NS: what its staged values leave room for)
  return NS && F64 ? 1 : (KG == 4 ? (NS ? 2 : (F64 ? 3 : (KU == 4 ? 4 : 5))) : 16 / KG);
}

// TS = storage of T_i (float / double), A = accumulation, F64 = record width
// NS: the NSNI stabilisation force rides along,
// f_J += sum_i sum_q W_i(k, q) S_q(i, J) (FINT.F90:1127-1208 layout), with the
// row weights W_i staged beside T_i.
// BODY: a body force (compiled apart: its sums and branches cost registers the
// plain step has no use for).
template <typename TS, typename A, bool F64, int KG, int KU, bool NS, bool BODY>
__global__ void __launch_bounds__(64 * KG, force_blocks<F64, KG, KU, NS>()) k_force_t(TiledForceArgs a) {
  extern __shared__ __align__(16) double smx[];
  __shared__ ColumnSums cs;
  const int64_t t = blockIdx.x;
  const int cnt = a.jcnt[t];
  const StagedT<TS, NS> sT(smx, cnt);
  const StageIds<KG> ids(a.jset + t * (int64_t)a.jmax, a.jmax);
  const int64_t c0 = t * a.R;
  const int slot = threadIdx.x / KG;
  const int64_t J = c0 + a.sv.ord[c0 + slot];
  const int q = threadIdx.x & (KG - 1);
  const unsigned gmask = group_mask<KG>();
  const bool valid = J < a.n;
  // this lane's first KU packed records are requested before the staging,
  // so their latency overlaps it
  if (!NS && !F64 && a.sv.ahead) prefetch_rest<F64, KG>(a.pk, a.sv, c0, slot, KU);
  const RowWalk<KG> walk(a.sv, c0, slot, q);
  const int nit = valid ? walk.nit : 0;
  constexpr bool kPipe = !NS && (!F64 || KU <= 2);
  int64_t p0 = 0, pend = 0;  // list positions, for the values that stay in list order
  if (valid && BODY) {
    p0 = a.colptr[J] + q;
    pend = a.colptr[J + 1];
  }
  Rec<F64> cur[KU];
  SRec<F64> csr[NS ? KU : 1];
  bool have = nit >= KU;
  if (have) {
#pragma unroll
    for (int u = 0; u < KU; ++u) {
      load_rec(a.pk, a.sv.nrec, walk.at(u), cur[u]);
      if constexpr (NS) csr[u].load(a.ns_scol, a.sv.nrec, walk.at(u));
    }
  }
  grid_wait();
  sT.template fill<BODY>(a, ids, cnt);
  prefetch_columns(a, c0);
  __syncthreads();
  if (valid) {
    A f0 = A(0), f1 = A(0), f2 = A(0);
    double e0 = 0.0, e1 = 0.0, e2 = 0.0;
    auto body = [&](int it, const Rec<F64>& rec, const SRec<F64>& sr) {
      const A g0 = (A)rec.x(), g1 = (A)rec.y(), g2 = (A)rec.z();
      const int l = rec.l();
      TS T[StagedT<TS, NS>::N];
      sT.t.load(l, T);
      f0 += (A)T[0] * g0 + (A)T[1] * g1 + (A)T[2] * g2;
      f1 += (A)T[3] * g0 + (A)T[4] * g1 + (A)T[5] * g2;
      f2 += (A)T[6] * g0 + (A)T[7] * g1 + (A)T[8] * g2;
      if constexpr (NS) {
        A sq[6];
        sr.get(sq);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          f0 += (A)StagedT<TS, NS>::weight(T, c) * sq[c];
          f1 += (A)StagedT<TS, NS>::weight(T, 6 + c) * sq[c];
          f2 += (A)StagedT<TS, NS>::weight(T, 12 + c) * sq[c];
        }
      }
      if (BODY) {
        const int64_t e = p0 + (int64_t)KG * it;
        if (e < pend) {  // (not a pad)
          const double s = a.tshp[e];
          double b[3];
          sT.body_of(a, l, b);
          e0 += s * b[0]; e1 += s * b[1]; e2 += s * b[2];
        }
      }
    };
    int it = 0;
    while (have) {  // as in the row gather
      const bool hn = it + 2 * KU <= nit;
      Rec<F64> nxt[KU];
      if constexpr (kPipe) {
#pragma unroll
        for (int u = 0; u < KU; ++u) {
          if (hn) load_rec(a.pk, a.sv.nrec, walk.at(it + KU + u), nxt[u]);
          else nxt[u] = cur[u];
        }
      }
#pragma unroll
      for (int u = 0; u < KU; ++u) body(it + u, cur[u], csr[NS ? u : 0]);
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        if constexpr (kPipe) {
          cur[u] = nxt[u];
        } else if (hn) {
          load_rec(a.pk, a.sv.nrec, walk.at(it + KU + u), cur[u]);
          if constexpr (NS) csr[u].load(a.ns_scol, a.sv.nrec, walk.at(it + KU + u));
        }
      }
      it += KU;
      have = hn;
    }
    for (; it < nit; ++it) {
      Rec<F64> rec;
      load_rec(a.pk, a.sv.nrec, walk.at(it), rec);
      SRec<F64> sr;
      if constexpr (NS) sr.load(a.ns_scol, a.sv.nrec, walk.at(it));
      body(it, rec, sr);
    }
#pragma unroll
    for (int o = 1; o < KG; o <<= 1) {
      f0 += __shfl_xor_sync(gmask, f0, o);
      f1 += __shfl_xor_sync(gmask, f1, o);
      f2 += __shfl_xor_sync(gmask, f2, o);
      if (BODY) {
        e0 += __shfl_xor_sync(gmask, e0, o);
        e1 += __shfl_xor_sync(gmask, e1, o);
        e2 += __shfl_xor_sync(gmask, e2, o);
      }
    }
    if (q < 3) {
      const int m = 3 * (int)(J - c0) + q;
      cs.f[m] = (double)(q == 0 ? f0 : (q == 1 ? f1 : f2));
      if (BODY) cs.e[m] = q == 0 ? e0 : (q == 1 ? e1 : e2);
    }
  }
  finish_columns<BODY>(a, c0, cs, 0u);
}

// ---- record streams through the copy engine ------------------------------
// The variants below ask the copy engine (cp.async.bulk) for the tile's
// whole record range, in kChunks chunks with an mbarrier each, before the
// block stages its neighbour data: the records stream into shared memory
// while the threads gather, and the entry loop then reads them from shared
// memory.  Sources are this GPU's record arrays (no peer memory, no
// multicast).  Every wait is bounded; a wait that gives up raises
// MEGA_ST_WAIT_TIMEOUT and the lane skips its sums.
constexpr int kChunks = 4;
constexpr int kPollLimit = 1 << 16;

// Thread 0: the barriers, then the copies of steps [0, ne) of the tile (32
// records each) from the record planes (16-byte records, or the 16-, 8- and
// 2-byte planes of FP64) into rec, where each plane has room for recmax
// records.
template <bool F64>
__device__ __forceinline__ void issue_records(uint64_t* bar, unsigned char* rec, const void* pk, int64_t nrec,
                                              int64_t step0, int64_t ne, int64_t recmax) {
  if (threadIdx.x != 0) return;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) mbar_init(&bar[c], 1);
  mbar_fence_init();
  constexpr int width[3] = {16, 8, 2};
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int64_t lo = c * ne / kChunks, hi = (c + 1) * ne / kChunks;
    mbar_arrive_expect(&bar[c], (uint32_t)((hi - lo) * 32 * (F64 ? 26 : 16)));
    const unsigned char* src = (const unsigned char*)pk;
    unsigned char* dst = rec;
#pragma unroll
    for (int k = 0; k < (F64 ? 3 : 1); ++k) {
      const uint32_t bytes = (uint32_t)((hi - lo) * 32 * width[k]);
      for (uint32_t off = 0; off < bytes; off += 32768u)
        bulk_load(dst + lo * 32 * width[k] + off, src + (step0 + lo) * 32 * width[k] + off,
                  min(32768u, bytes - off), &bar[c]);
      src += nrec * width[k];
      dst += recmax * width[k];
    }
  }
}

// Wait for the chunks holding steps [a, b) of the tile.
__device__ __forceinline__ bool wait_records(uint64_t* bar, int64_t ne, int64_t a, int64_t b) {
  bool ok = true;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int64_t lo = c * ne / kChunks, hi = (c + 1) * ne / kChunks;
    if (ok && lo < b && hi > a) ok = mbar_wait_bounded(&bar[c], 0, kPollLimit);
  }
  return ok;
}

// Thread 0 before the block retires: no copy of the block is left in flight.
__device__ __forceinline__ void drain_records(uint64_t* bar) {
  if (threadIdx.x != 0) return;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) mbar_wait_bounded(&bar[c], 0, kPollLimit);
}

// a staged record of the tile (planes of recmax records)
__device__ __forceinline__ void staged_rec(const unsigned char* rec, int64_t, int64_t p, Rec<false>& o) {
  o.v = reinterpret_cast<const float4*>(rec)[p];
}
__device__ __forceinline__ void staged_rec(const unsigned char* rec, int64_t recmax, int64_t p, Rec<true>& o) {
  const double2* xy = reinterpret_cast<const double2*>(rec);
  const double* z = reinterpret_cast<const double*>(xy + recmax);
  o.a = xy[p];
  o.b = z[p];
  o.r = reinterpret_cast<const uint16_t*>(z + recmax)[p];
}

// (the increments alone: FULL steps take the register kernel)
template <typename A, bool F64, bool INTERP, int KG>
__global__ void __launch_bounds__(64 * KG)
    k_defgrad_b(int32_t n, int32_t R, int32_t jmax, int32_t recmax, SliceView sv, const int64_t* __restrict__ rowptr,
                const void* __restrict__ pk, const int32_t* __restrict__ jset, const int32_t* __restrict__ jcnt,
                const double* dsp, const double* __restrict__ sdphi, const double* __restrict__ shp,
                double* dsp_tot_phy, double* fg, StepAccum* acc, unsigned* status) {
  constexpr int RB = F64 ? 26 : 16;
  extern __shared__ __align__(128) unsigned char smb[];
  __shared__ uint64_t bar[kChunks];
  const int64_t t = blockIdx.x;
  const int64_t r0 = t * R;
  const int64_t e0 = sv.sstep[r0 >> 3], ne = sv.sstep[(r0 + R) >> 3] - e0;
  issue_records<F64>(bar, smb, pk, sv.nrec, e0, ne, recmax);
  const int cnt = jcnt[t];
  const StageIds<KG> ids(jset + t * (int64_t)jmax, jmax);
  using SV = typename DispStage<F64>::V;
  constexpr int SN = DispStage<F64>::N;
  const Staged<SV, SN> sd{reinterpret_cast<SV*>(smb + (size_t)recmax * RB), staged_ld(cnt)};
  const int slot = threadIdx.x / KG;
  const int64_t i = r0 + sv.ord[r0 + slot];
  const int q = threadIdx.x & (KG - 1);
  const unsigned gmask = group_mask<KG>();
  const bool valid = i < n;
  grid_wait();
  if (acc && blockIdx.x == 0 && threadIdx.x < 32) clear_counts(acc);
  double dr[3] = {0.0, 0.0, 0.0};
  if (!F64) {
#pragma unroll
    for (int k = 0; k < 3; ++k) dr[k] = dsp[3 * r0 + k];
  }
  stage_disp<F64, KG>(ids, cnt, dsp, dr, sd);
  __syncthreads();
  if (valid) {
    const int64_t sl = (r0 + slot) >> 3;
    const bool ok = __all_sync(gmask, wait_records(bar, ne, sv.sstep[sl] - e0, sv.sstep[sl + 1] - e0));
    const RowWalk<KG> walk(sv, r0, slot, q);
    int64_t p0 = 0, pend = 0;
    if (INTERP) {
      p0 = rowptr[i] + q;
      pend = rowptr[i + 1];
    }
    double di[3];
    A fd[3], L[9];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      di[k] = dsp[3 * i + k];
      fd[k] = F64 ? (A)di[k] : (A)(float)(di[k] - dr[k]);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) L[k] = A(0);
    double ph[3] = {0.0, 0.0, 0.0};
    if (ok) {
#pragma unroll 4
      for (int it = 0; it < walk.nit; ++it) {
        Rec<F64> rec;
        staged_rec(smb, recmax, walk.at(it) - 32 * e0, rec);
        const A g[3] = {(A)rec.x(), (A)rec.y(), (A)rec.z()};
        const int l = rec.l();
        SV v[SN];
        sd.load(l, v);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const A d = (A)v[k] - fd[k];
          L[3 * k] += d * g[0]; L[3 * k + 1] += d * g[1]; L[3 * k + 2] += d * g[2];
        }
        if (INTERP) {
          const int64_t p = p0 + (int64_t)KG * it;
          if (p < pend) {
            const double s = shp[p];
#pragma unroll
            for (int k = 0; k < 3; ++k) ph[k] += s * (F64 ? (double)v[k] : dr[k] + (double)v[k]);
          }
        }
      }
    }
#pragma unroll
    for (int o = 1; o < KG; o <<= 1) {
#pragma unroll
      for (int k = 0; k < 9; ++k) L[k] += __shfl_xor_sync(gmask, L[k], o);
      if (INTERP) {
#pragma unroll
        for (int k = 0; k < 3; ++k) ph[k] += __shfl_xor_sync(gmask, ph[k], o);
      }
    }
    if (q == 0) {
      if (!ok) {
        atomicOr(status, (unsigned)MEGA_ST_WAIT_TIMEOUT);
      } else {
        const double sd3[3] = {sdphi[3 * i], sdphi[3 * i + 1], sdphi[3 * i + 2]};
        double h[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) h[k] = (double)L[k] + di[k / 3] * sd3[k % 3];
        store_g0(fg, fg_ld(n), i, !F64, h);
        if (INTERP) {
#pragma unroll
          for (int k = 0; k < 3; ++k) dsp_tot_phy[3 * i + k] += ph[k];
        }
      }
    }
  }
  drain_records(bar);
}

template <typename TS, typename A, bool F64, int KG>
__global__ void __launch_bounds__(64 * KG) k_force_b(TiledForceArgs a) {
  constexpr int RB = F64 ? 26 : 16;
  extern __shared__ __align__(128) unsigned char smb[];
  __shared__ uint64_t bar[kChunks];
  __shared__ ColumnSums cs;
  const int64_t t = blockIdx.x;
  const int64_t c0 = t * a.R;
  const int64_t e0 = a.sv.sstep[c0 >> 3], ne = a.sv.sstep[(c0 + a.R) >> 3] - e0;
  issue_records<F64>(bar, smb, a.pk, a.sv.nrec, e0, ne, a.recmax);
  const int cnt = a.jcnt[t];
  const StagedT<TS, false> sT(smb + (size_t)a.recmax * RB, cnt);
  const StageIds<KG> ids(a.jset + t * (int64_t)a.jmax, a.jmax);
  const int slot = threadIdx.x / KG;
  const int64_t J = c0 + a.sv.ord[c0 + slot];
  const int q = threadIdx.x & (KG - 1);
  const unsigned gmask = group_mask<KG>();
  const bool valid = J < a.n;
  grid_wait();
  if (a.has_body) sT.template fill<true>(a, ids, cnt);
  else sT.template fill<false>(a, ids, cnt);
  prefetch_columns(a, c0);
  __syncthreads();
  unsigned st = 0;
  if (valid) {
    const int64_t sl = (c0 + slot) >> 3;
    const bool ok = __all_sync(gmask, wait_records(bar, ne, a.sv.sstep[sl] - e0, a.sv.sstep[sl + 1] - e0));
    const RowWalk<KG> walk(a.sv, c0, slot, q);
    int64_t p0 = 0, pend = 0;
    if (a.has_body) {
      p0 = a.colptr[J] + q;
      pend = a.colptr[J + 1];
    }
    A f0 = A(0), f1 = A(0), f2 = A(0);
    double b0 = 0.0, b1 = 0.0, b2 = 0.0;
    if (ok) {
#pragma unroll 4
      for (int it = 0; it < walk.nit; ++it) {
        Rec<F64> rec;
        staged_rec(smb, a.recmax, walk.at(it) - 32 * e0, rec);
        const A g0 = (A)rec.x(), g1 = (A)rec.y(), g2 = (A)rec.z();
        const int l = rec.l();
        TS T[9];
        sT.t.load(l, T);
        f0 += (A)T[0] * g0 + (A)T[1] * g1 + (A)T[2] * g2;
        f1 += (A)T[3] * g0 + (A)T[4] * g1 + (A)T[5] * g2;
        f2 += (A)T[6] * g0 + (A)T[7] * g1 + (A)T[8] * g2;
        if (a.has_body) {
          const int64_t p = p0 + (int64_t)KG * it;
          if (p < pend) {
            const double s = a.tshp[p];
            double b[3];
            sT.body_of(a, l, b);
            b0 += s * b[0]; b1 += s * b[1]; b2 += s * b[2];
          }
        }
      }
    }
#pragma unroll
    for (int o = 1; o < KG; o <<= 1) {
      f0 += __shfl_xor_sync(gmask, f0, o);
      f1 += __shfl_xor_sync(gmask, f1, o);
      f2 += __shfl_xor_sync(gmask, f2, o);
      if (a.has_body) {
        b0 += __shfl_xor_sync(gmask, b0, o);
        b1 += __shfl_xor_sync(gmask, b1, o);
        b2 += __shfl_xor_sync(gmask, b2, o);
      }
    }
    if (!ok && q == 0) st |= MEGA_ST_WAIT_TIMEOUT;  // (the step's outputs are void)
    if (q < 3) {
      const int m = 3 * (int)(J - c0) + q;
      cs.f[m] = (double)(q == 0 ? f0 : (q == 1 ? f1 : f2));
      if (a.has_body) cs.e[m] = q == 0 ? b0 : (q == 1 ? b1 : b2);
    }
  }
  if (a.has_body) finish_columns<true>(a, c0, cs, st);
  else finish_columns<false>(a, c0, cs, st);
  drain_records(bar);
}

inline unsigned grid_for(int64_t work, int block) { return (unsigned)((work + block - 1) / block); }

}  // namespace

int build_tiles(cudaStream_t s, int32_t n, const int64_t* ptr, const int32_t* idx, int64_t nnz, int32_t gmaxn,
                TileSet& ts, DevPool& pool, int32_t* maxcnt_out, int32_t rows) {
  constexpr int HS = 2048;
  const int32_t jmax = HS / 2;
  if (gmaxn > jmax) return MEGA_ERR_UNSUPPORTED;
  DevPool scratch(s);
  int16_t* slot_tmp = nullptr;
  int32_t* ovf = nullptr;
  MEGA_ALLOC(scratch, slot_tmp, nnz);
  MEGA_ALLOC(scratch, ovf, 1);
  for (int32_t R = rows; R >= 8; R >>= 1) {  // >= 8 keeps every block a whole warp
    const int64_t ntiles = (n + R - 1) / R;
    int32_t *jset = nullptr, *jcnt = nullptr;
    uint16_t* lidx = nullptr;
    DevPool trial;
    if (pool.ordered) trial.bind(pool.stream);
    MEGA_ALLOC(trial, jset, ntiles * jmax);
    MEGA_ALLOC(trial, jcnt, ntiles);
    MEGA_ALLOC(trial, lidx, nnz);
    MEGA_TRY(cudaMemsetAsync(ovf, 0, sizeof(int32_t), s));
    k_build_tiles<HS><<<(unsigned)ntiles, 256, 0, s>>>(n, R, ptr, idx, jmax, jset, jcnt, lidx, slot_tmp, ovf);
    MEGA_CHECK_LAUNCH();
    int32_t hovf = 0;
    MEGA_TRY(cudaMemcpyAsync(&hovf, ovf, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    std::vector<int32_t> hc(ntiles);
    MEGA_TRY(cudaMemcpyAsync(hc.data(), jcnt, sizeof(int32_t) * ntiles, cudaMemcpyDeviceToHost, s));
    MEGA_TRY(cudaStreamSynchronize(s));
    if (hovf) continue;  // too many distinct neighbours: halve the tile
    int32_t mx = 0;
    for (int32_t v : hc) mx = std::max(mx, v);
    // keep the trial buffers: move ownership into the persistent pool
    pool.adopt(trial);
    ts.R = R;
    ts.ntiles = ntiles;
    ts.jmax = jmax;
    ts.maxcnt = mx;
    ts.jset = jset;
    ts.jcnt = jcnt;
    ts.lidx = lidx;
    if (maxcnt_out) *maxcnt_out = mx;
    return 0;
  }
  return MEGA_ERR_UNSUPPORTED;
}

int build_slices(cudaStream_t s, int32_t n, const int64_t* ptr, TileSet& ts, DevPool& pool) {
  const int64_t slots = ts.ntiles * ts.R, nsl = slots / 8;
  DevPool scratch(s);
  int32_t *steps = nullptr, *most = nullptr;
  MEGA_ALLOC(scratch, steps, nsl);
  MEGA_ALLOC(scratch, most, 1);
  MEGA_ALLOC(pool, ts.ord, slots);
  MEGA_ALLOC(pool, ts.sstep, nsl + 1);
  MEGA_ALLOC(pool, ts.rbase, n);
  MEGA_TRY(cudaMemsetAsync(most, 0, sizeof(int32_t), s));
  k_slice_rows<<<(unsigned)ts.ntiles, 64, 0, s>>>(n, ts.R, ptr, ts.ord, steps, most);
  MEGA_CHECK_LAUNCH();
  if (int r = scan_counts(s, steps, ts.sstep, nsl, scratch)) return r;
  k_slice_base<<<grid_for(slots, 256), 256, 0, s>>>(n, ts.R, slots, ts.ord, ts.sstep, ts.rbase);
  MEGA_CHECK_LAUNCH();
  int64_t total = 0;
  int32_t tile = 0;
  MEGA_TRY(cudaMemcpyAsync(&total, ts.sstep + nsl, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  MEGA_TRY(cudaMemcpyAsync(&tile, most, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  MEGA_TRY(cudaStreamSynchronize(s));
  ts.nrec = 32 * total;
  ts.recmax = 32 * tile;
  return 0;
}

int pack_transposed32(cudaStream_t s, int32_t n, const TileSet& ct, const int64_t* colptr, const float4* in,
                      const int32_t* trow, const int64_t* pos, const int64_t* rowptr, const TileSet& rt,
                      float4* out) {
  const int64_t slots = ct.ntiles * ct.R;
  k_pack_t32<<<grid_for(4 * slots, 256), 256, 0, s>>>(n, ct.R, slots, ct.view(), colptr, ct.lidx, in, trow, pos,
                                                      rowptr, rt.rbase, out);
  MEGA_CHECK_LAUNCH();
  return 0;
}

int pack_entries(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, const double* gx,
                 const double* gy, const double* gz, const int64_t* pos, bool f64, void* out) {
  const int64_t slots = ts.ntiles * ts.R;
  const unsigned grid = grid_for(4 * slots, 256);
  if (f64) k_pack_f64<<<grid, 256, 0, s>>>(n, ts.R, slots, ts.view(), ptr, ts.lidx, gx, gy, gz, pos, out);
  else k_pack_f32<<<grid, 256, 0, s>>>(n, ts.R, slots, ts.view(), ptr, ts.lidx, gx, gy, gz, pos, (float4*)out);
  MEGA_CHECK_LAUNCH();
  return 0;
}

int pad_records32(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, float4* out) {
  const int64_t slots = ts.ntiles * ts.R;
  k_pad_f32<<<grid_for(4 * slots, 256), 256, 0, s>>>(n, ts.R, slots, ts.view(), ptr, ts.lidx, out);
  MEGA_CHECK_LAUNCH();
  return 0;
}

int bank_order(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, uint16_t* lidx,
               int64_t* pos, int lanes) {
  if (n <= 0) return 0;
  if ((lanes != 4 && lanes != 8) || ts.R * lanes < 32) return MEGA_ERR_UNSUPPORTED;
  const int64_t nwarps = ts.ntiles * (int64_t)(ts.R * lanes / 32);
  const unsigned grid = (unsigned)((nwarps * 32 + 127) / 128);
  if (lanes == 4) k_bank_order<4, 8, 8><<<grid, 128, 0, s>>>(n, ts.R, nwarps, ts.ord, ptr, lidx, pos);
  else k_bank_order<8, 8, 8><<<grid, 128, 0, s>>>(n, ts.R, nwarps, ts.ord, ptr, lidx, pos);
  MEGA_CHECK_LAUNCH();
  return 0;
}

int iota64(cudaStream_t s, int64_t m, int64_t* out) {
  if (m <= 0) return 0;
  k_iota64<<<grid_for(m, 256), 256, 0, s>>>(m, out);
  MEGA_CHECK_LAUNCH();
  return 0;
}

int pack_second(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, const int64_t* pos, const NsniS& src,
                bool f64, void* out) {
  const int64_t slots = ts.ntiles * ts.R;
  auto k = f64 ? k_pack_second<true> : k_pack_second<false>;
  k<<<grid_for(4 * slots, 256), 256, 0, s>>>(n, ts.R, slots, ts.view(), ptr, pos, src, out);
  MEGA_CHECK_LAUNCH();
  return 0;
}

int gather_second(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, const int64_t* pos, bool f64,
                  const void* in, void* out) {
  const int64_t slots = ts.ntiles * ts.R;
  auto k = f64 ? k_gather_second<true> : k_gather_second<false>;
  k<<<grid_for(4 * slots, 256), 256, 0, s>>>(n, ts.R, slots, ts.view(), ptr, pos, in, out);
  MEGA_CHECK_LAUNCH();
  return 0;
}

int gather_records(cudaStream_t s, int32_t n, const TileSet& ts, const int64_t* ptr, const int64_t* pos, bool f64,
                   const void* in, void* out) {
  const int64_t slots = ts.ntiles * ts.R;
  const unsigned grid = grid_for(4 * slots, 256);
  if (f64) k_gather_rec64<<<grid, 256, 0, s>>>(n, ts.R, slots, ts.view(), ptr, pos, in, out);
  else k_gather_rec32<<<grid, 256, 0, s>>>(n, ts.R, slots, ts.view(), ptr, pos, (const float4*)in, (float4*)out);
  MEGA_CHECK_LAUNCH();
  return 0;
}

// The launch variants, in the order the autotuner tries them:
// (KG, KU) = (4, 4), (4, 2), (4, 1), (8, 2) with register-held record
// streams, then KG = 4, 8 with the records streamed into shared memory, then
// (16, 1), (16, 2) with register-held streams (four times the threads per
// staged neighbour of KG = 4: the NSNI force gather stages 27 values a node).
constexpr int kVariants = kTiledVariants;
// records in flight per lane of the FULL gathers (one step in 16: one form
// per lane count; the count in flight does not change a row's sum)
constexpr int kFullKU = 2;
// dynamic shared memory a streamed-variant block may ask for: sm_100's 227 KB
// per block less room for the kernels' static shared memory (under 1 KB)
constexpr int kBulkSmemMax = 227 * 1024 - 1024;

// The dynamic shared-memory limit is raised, to the same value by every caller,
// only for a launch that may pass 48 KB with the kernel's static part (4 KB at
// most): raising it for every kernel at set-up loaded all of them (20 ms of a
// process's first search).  load_only does both ahead of a stream capture.
template <typename K>
static int raise_smem(K k, int lim) {
  MEGA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  return 0;
}
template <typename... KA, typename... A>
static int start(void (*k)(KA...), int lim, bool load_only, unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                 A&&... args) {
  if (smem > 44 * 1024)
    if (int r = raise_smem(k, lim)) return r;
  if (load_only) {
    cudaFuncAttributes fa{};
    MEGA_TRY(cudaFuncGetAttributes(&fa, k));
    return 0;
  }
  return launch_overlapped(k, grid, block, smem, s, std::forward<A>(args)...);
}
// A tile stages at most 1024 neighbours: 96 KB for the double-precision T_i of
// the column gather, 120 KB for the float T_i and NSNI weights.
static int stage_limit() { return 31 * 4 * staged_ld(1024); }

// what the streamed variants may ask for: the device's limit less the kernels'
// static shared memory, raised for all of them at the first question
static int g_bulk_lim = kBulkSmemMax;

template <typename K>
static int raise_smem_upto(K k, int lim) {
  cudaFuncAttributes fa{};
  MEGA_TRY(cudaFuncGetAttributes(&fa, k));
  const int room = lim - (int)fa.sharedSizeBytes;
  g_bulk_lim = std::min(g_bulk_lim, room);
  return raise_smem(k, room);
}

template <int KG>
static int configure_bulk(int lim) {
  int dev = 0, optin = 0;
  MEGA_TRY(cudaGetDevice(&dev));
  MEGA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  lim = std::min(lim + 1024, optin);  // the kernels' static shared memory comes off this
  int r = 0;
  if ((r = raise_smem_upto(k_defgrad_b<float, false, true, KG>, lim))) return r;
  if ((r = raise_smem_upto(k_defgrad_b<float, false, false, KG>, lim))) return r;
  if ((r = raise_smem_upto(k_defgrad_b<double, true, true, KG>, lim))) return r;
  if ((r = raise_smem_upto(k_defgrad_b<double, true, false, KG>, lim))) return r;
  if ((r = raise_smem_upto(k_force_b<float, float, false, KG>, lim))) return r;
  return raise_smem_upto(k_force_b<double, double, true, KG>, lim);
}

static bool bulk_fits(size_t smem) {
  static const int r = [] {
    const int a = configure_bulk<4>(kBulkSmemMax);
    return a ? a : configure_bulk<8>(kBulkSmemMax);
  }();
  return r == 0 && smem <= (size_t)g_bulk_lim;
}

int tiled_variants() { return kVariants; }

bool tiled_variant_fits(const TileSet& ts, bool mixed, int variant, bool force, bool has_body) {
  if (variant < 0 || variant >= kVariants) return false;
  if (variant < 4 || variant > 5) return true;  // register variants
  const size_t stage = force ? (mixed ? sizeof(float) : sizeof(double)) * (has_body ? 12 : 9) : (mixed ? 16 : 24);
  return bulk_fits((size_t)ts.recmax * (mixed ? 16 : 26) + stage * staged_ld(ts.maxcnt));
}

// one launch's arguments of the row gather
struct DefgradArgs {
  bool mixed, interp;
  int32_t n;
  const TileSet& ts;
  const NsniTiles* ns;
  const int64_t* rowptr;
  const void* pk;
  const double *dsp, *dsp_tot, *sdphi, *shp;
  double *dsp_tot_phy, *fg;
  StepAccum* acc;
  unsigned* status;
  bool load_only;
};

template <int KG>
static int defgrad_bulk(cudaStream_t s, const DefgradArgs& d) {
  const TileSet& ts = d.ts;
  const size_t smem = (size_t)ts.recmax * (d.mixed ? 16 : 26) + (size_t)(d.mixed ? 16 : 24) * staged_ld(ts.maxcnt);
  if (!bulk_fits(smem)) return MEGA_ERR_UNSUPPORTED;
  auto k = d.mixed ? (d.interp ? k_defgrad_b<float, false, true, KG> : k_defgrad_b<float, false, false, KG>)
                   : (d.interp ? k_defgrad_b<double, true, true, KG> : k_defgrad_b<double, true, false, KG>);
  return start(k, g_bulk_lim, d.load_only, (unsigned)ts.ntiles, ts.R * KG, smem, s, d.n, ts.R, ts.jmax, ts.recmax,
               ts.view(), d.rowptr, d.pk, ts.jset, ts.jcnt, d.dsp, d.sdphi, d.shp, d.dsp_tot_phy, d.fg, d.acc, d.status);
}

template <int KG, int KU, bool FULL = false>
static int defgrad_variant(cudaStream_t s, const DefgradArgs& d) {
  const TileSet& ts = d.ts;
  const size_t smem = (size_t)((d.mixed ? 16 : 24) * (FULL ? 2 : 1)) * staged_ld(ts.maxcnt);
  const NsniTiles nz = d.ns ? *d.ns : NsniTiles();
  auto k = !d.mixed ? (d.ns ? (d.interp ? k_defgrad_t<double, true, true, KG, KU, true, FULL>
                                        : k_defgrad_t<double, true, false, KG, KU, true, FULL>)
                            : (d.interp ? k_defgrad_t<double, true, true, KG, KU, false, FULL>
                                        : k_defgrad_t<double, true, false, KG, KU, false, FULL>))
           : d.ns   ? (d.interp ? k_defgrad_t<float, false, true, KG, KU, true, FULL>
                                : k_defgrad_t<float, false, false, KG, KU, true, FULL>)
                    : (d.interp ? k_defgrad_t<float, false, true, KG, KU, false, FULL>
                                : k_defgrad_t<float, false, false, KG, KU, false, FULL>);
  return start(k, stage_limit(), d.load_only, (unsigned)ts.ntiles, ts.R * KG, smem, s, d.n, ts.R, ts.jmax, nz,
               ts.view(records_ahead(ts, d.mixed)),
               d.rowptr, d.pk, ts.jset, ts.jcnt, d.dsp, d.dsp_tot, d.sdphi, d.shp, d.dsp_tot_phy, d.fg, d.acc, NoStress());
}

// NSNI runs the register variants: mixed refuses the streamed ones, FP64 takes
// the register variant of the same lanes per row (the same sums) for them.
static bool ns_variant(bool mixed, int& variant) {
  if (variant != 4 && variant != 5) return true;
  variant = variant == 4 ? 0 : 3;
  return !mixed;
}

int launch_defgrad_tiled(cudaStream_t s, bool mixed, bool interp, int32_t n, const TileSet& ts,
                         const NsniTiles* ns, const int64_t* rowptr, const void* pk, const double* dsp,
                         const double* dsp_tot, const double* sdphi, const double* shp, double* dsp_tot_phy,
                         double* fg, StepAccum* acc, unsigned* status, int variant, bool full, bool load_only) {
  int r = 0;
  if (ns && !ns_variant(mixed, variant)) return MEGA_ERR_UNSUPPORTED;
  const DefgradArgs d{mixed, interp, n, ts, ns, rowptr, pk, dsp, dsp_tot, sdphi, shp, dsp_tot_phy, fg, acc, status,
                      load_only};
  if (full) {
    if (variant == 6 || variant == 7) r = defgrad_variant<16, kFullKU, true>(s, d);
    else if (variant == 3 || variant == 5) r = defgrad_variant<8, kFullKU, true>(s, d);
    else r = defgrad_variant<4, kFullKU, true>(s, d);
  } else {
    switch (variant) {
      case 1: r = defgrad_variant<4, 2>(s, d); break;
      case 2: r = defgrad_variant<4, 1>(s, d); break;
      case 3: r = defgrad_variant<8, 2>(s, d); break;
      case 4: r = defgrad_bulk<4>(s, d); break;
      case 5: r = defgrad_bulk<8>(s, d); break;
      case 6: r = defgrad_variant<16, 1>(s, d); break;
      case 7: r = defgrad_variant<16, 2>(s, d); break;
      default: r = defgrad_variant<4, 4>(s, d);
    }
  }
  if (r) return r;
  MEGA_CHECK_LAUNCH();
  return 0;
}

template <int KG, int KU>
static int defgrad_stress(cudaStream_t s, const DefgradArgs& d, const StressArgs& a) {
  const TileSet& ts = d.ts;
  const size_t smem = (size_t)(d.mixed ? 16 : 24) * staged_ld(ts.maxcnt);
  auto k = d.mixed ? k_defgrad_t<float, false, false, KG, KU, false, false, StressArgs>
                   : k_defgrad_t<double, true, false, KG, KU, false, false, StressArgs>;
  return start(k, stage_limit(), d.load_only, (unsigned)ts.ntiles, ts.R * KG, smem, s, d.n, ts.R, ts.jmax, NsniTiles(),
               ts.view(records_ahead(ts, d.mixed)), d.rowptr, d.pk, ts.jset, ts.jcnt, d.dsp, d.dsp_tot, d.sdphi, d.shp, d.dsp_tot_phy, d.fg, d.acc,
               a);
}

// Fetched ahead where a gather's blocks are all resident at once, so that only
// their own latency counts (steps of 4,455 nodes, FP64 17.3 -> 16.5 us, mixed 13.3
// -> 12.5; FP64 in the joined row gather alone), and mixed where the bank-ordered
// records of both gathers pass the L2 three times, so that they come from HBM
// (1.04 M nodes 601 -> 576; 255 k, four times the L2, 168 -> 164).  In between part
// of them is still in L2 and the requests only take its bandwidth (130 k nodes,
// twice the L2, 88 -> 93; FP64 135 -> 148); in list order the gathers wait for bank
// conflicts instead (383 k 250 -> 253).
bool records_ahead(const TileSet& ts, bool mixed) {
  static const int64_t l2 = [] {
    int dev = 0, bytes = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&bytes, cudaDevAttrL2CacheSize, dev) != cudaSuccess || bytes <= 0)
      bytes = 126 << 20;
    return (int64_t)bytes;
  }();
  return ts.ntiles <= 2 * (int64_t)device_sm_count() || (mixed && ts.banked32 && 2 * 16 * ts.nrec > 3 * l2);
}

// Joined where every block is resident at once (two of 256 threads an SM, one
// of 512): joined and apart, 4,455 nodes FP64 16.6 and 18.3 us a step, 16,154 24.9
// and 27.3; past the line the update's registers cost the gather its warps, 23,782
// nodes 38.8 and 34.4 (mixed alike).
bool defgrad_stress_fits(const TileSet& ts, int variant) {
  const int lanes = variant >= 6 ? 16 : (variant == 3 || variant == 5 ? 8 : 4);
  const int threads = ts.R * lanes;
  return threads <= 512 && ts.ntiles <= (int64_t)device_sm_count() * (512 / threads > 2 ? 2 : 512 / threads);
}

int launch_defgrad_stress(cudaStream_t s, bool mixed, int32_t n, const TileSet& ts, const int64_t* rowptr,
                          const void* pk, const double* dsp, const double* dsp_tot, const double* sdphi, double* fg,
                          const StressArgs& a, int variant, bool load_only) {
  const DefgradArgs d{mixed, false, n,      ts,   nullptr, rowptr, pk, dsp, dsp_tot, sdphi, nullptr, nullptr, fg,
                      a.acc, a.status, load_only};
  if (variant >= 6) return defgrad_stress<16, 2>(s, d, a);
  if (variant == 3 || variant == 5) return defgrad_stress<8, 2>(s, d, a);
  return defgrad_stress<4, 4>(s, d, a);
}

template <int KG>
static int force_bulk(cudaStream_t s, bool mixed, const TiledForceArgs& a, bool load_only) {
  const int nv = a.has_body ? 12 : 9;
  const size_t smem = (size_t)a.recmax * (mixed ? 16 : 26) + (mixed ? sizeof(float) : sizeof(double)) * nv *
                      staged_ld(a.maxcnt);
  if (!bulk_fits(smem)) return MEGA_ERR_UNSUPPORTED;
  const unsigned grid = (unsigned)a.ntiles;
  const int block = a.R * KG;
  return start(mixed ? k_force_b<float, float, false, KG> : k_force_b<double, double, true, KG>, g_bulk_lim, load_only,
               grid, block, smem, s, a);
}

template <int KG, int KU, bool BODY>
static auto force_kernel(bool mixed, bool ns) {
  return !mixed ? (ns ? k_force_t<double, double, true, KG, KU, true, BODY> : k_force_t<double, double, true, KG, KU, false, BODY>)
                : (ns ? k_force_t<float, float, false, KG, KU, true, BODY> : k_force_t<float, float, false, KG, KU, false, BODY>);
}

template <int KG, int KU>
static int force_variant(cudaStream_t s, bool mixed, const TiledForceArgs& a, bool load_only) {
  const size_t smem = !mixed ? (a.ns_scol ? StagedT<double, true>::bytes(a.maxcnt, a.has_body)
                                          : StagedT<double, false>::bytes(a.maxcnt, a.has_body))
                             : (a.ns_scol ? StagedT<float, true>::bytes(a.maxcnt, a.has_body)
                                          : StagedT<float, false>::bytes(a.maxcnt, a.has_body));
  const unsigned grid = (unsigned)a.ntiles;
  const int block = a.R * KG;
  auto k = force_kernel<KG, KU, false>(mixed, a.ns_scol != nullptr);
  if (a.has_body) k = force_kernel<KG, KU, true>(mixed, a.ns_scol != nullptr);
  const int lim = !mixed && a.ns_scol ? (int)StagedT<double, true>::bytes(1024, true) : stage_limit();
  return start(k, lim, load_only, grid, block, smem, s, a);
}

int launch_force_tiled(cudaStream_t s, bool mixed, const TiledForceArgs& a, int variant, bool load_only) {
  int r = 0;
  if (a.ns_scol && !ns_variant(mixed, variant)) return MEGA_ERR_UNSUPPORTED;
  switch (variant) {
    case 1: r = force_variant<4, 2>(s, mixed, a, load_only); break;
    case 2: r = force_variant<4, 1>(s, mixed, a, load_only); break;
    case 3: r = force_variant<8, 2>(s, mixed, a, load_only); break;
    case 6: r = force_variant<16, 1>(s, mixed, a, load_only); break;
    case 7: r = force_variant<16, 2>(s, mixed, a, load_only); break;
    case 4: r = force_bulk<4>(s, mixed, a, load_only); break;
    case 5: r = force_bulk<8>(s, mixed, a, load_only); break;
    default: r = force_variant<4, 4>(s, mixed, a, load_only);
  }
  if (r) return r;
  MEGA_CHECK_LAUNCH();
  return 0;
}

}  // namespace mega
