// Kernels of the SPH geomechanics step (sm_100a).  Layout in HBM: structure of
// arrays, one 16-byte (float) / 32-byte (double) vector per particle per field,
// particles sorted by cell key (boundary cells first, then material cells, then the
// deleted cell), so the 27 neighbour cells of a particle are 9 contiguous index runs
// per layer and neighbour reads of consecutive particles hit the same lines.
#pragma once
#include <float.h>
#include <limits.h>

#include "rw_device.cuh"
#include "rw_mlp.cuh"
#include "rw_params.h"

namespace rw {

// Per-particle record consumed by the pair loop of the interaction: everything the
// reference recomputes per neighbour pair from j's state (mass, volume, sigma/rho^2),
// computed once per particle per section.  48 bytes in float: the contact-wall flag
// travels as the sign of the (always positive) volume.
template <class T> struct Rec {
  V4<T> p;   // in-cell position (w unused): one aligned 64-byte record per neighbour in float
  V4<T> vr;  // velocity xyz, density
  V4<T> a;   // mass, +-volume (negative: contact-wall particle), sigma/rho^2 xx, yy
  V4<T> b;   // sigma/rho^2 zz, xy, xz, yz
};

template <class T> struct DevState {
  // Permuted every section (ping-pong, Dyn::cur_main selects the live buffer).
  int4* codes[2];
  int4* cellpos[2];
  V4<T>* pos[2];
  V4<T>* pos_ori[2];
  V4<T>* vel[2];
  V4<T>* idm[2];
  V4<T>* str_a[2];
  V2<T>* str_b[2];
  V4<T>* stn_a[2];
  V2<T>* stn_b[2];
  // Permuted in the predictor section only (SortArraysPrimary), Dyn::cur_nrm.
  V4<T>* normal[2];
  // Permuted in the corrector section only (SortArraysAll), Dyn::cur_ini.
  V4<T>* pos_ini[2];
  V4<T>* vel_ini[2];
  V4<T>* stri_a[2];
  V2<T>* stri_b[2];
  V4<T>* stni_a[2];
  V2<T>* stni_b[2];
  // Compensation terms of the precision form (position xyz, velocity xyz+rho),
  // permuted with the particles; *_ini copies saved by the predictor.
  V4<T>* cmp_p[2];
  V4<T>* cmp_v[2];
  V4<T>* cmp_pi[2];
  V4<T>* cmp_vi[2];
  // Stage outputs, indexed like the live buffers.
  V4<T>* accad;
  V4<T>* spin;
  V4<T>* ace_a;
  V2<T>* ace_b;
  // Contact state bound to array slots, as in the reference (never permuted there).
  // contact_var and the contact force are double-buffered across the interaction so
  // that every particle reads the others' values as of the start of the stage.
  V4<T>* cv[2];   // kernel integral, distance along normal, slide flag, wall id
  V4<T>* cf[2];   // contact force xyz
  V4<T>* cny;     // contact normal (contact_mag.yx..yz)
  V4<T>* cvz;     // contact velocity (contact_mag.zx..zz)
  Rec<T>* rec;
  V4<T>* tc_a;    // Shepard result (tensor2d_cache)
  V2<T>* tc_b;
  // Cell list.
  int* keys;      // cell key per particle (unsorted order)
  int* vals;
  int* tk;        // radix-sort ping-pong
  int* tv;
  const int* skeys;  // sorted keys / permutation (one of keys|tk, vals|tv)
  const int* sperm;
  int2* range;    // [beg, end) per cell, (0,0) when empty
  int* hist;      // radix-sort digit counts per tile
  int* dtot;      // per-digit totals
  int sort_passes;
  double* wsum;   // wall-force partial sums
  // Column chunks of the interaction (rebuilt after every sort).
  int* col_beg;
  int* col_len;
  int* col_cnt;
  int* col_off;
  struct Chunk* chunks;
  // Candidate lists of the soil particles, four entries to a quad (entry e of soil slot t at
  // nbg[b][(e / 4) * 4 * nbg_stride + 4 t + e % 4], the last quad filled up with an entry of
  // the particle itself), count per slot (-1: not kept).  Two buffers
  // b, Dyn::lbuf the live one: a list update after a permutation reads the other.
  unsigned* nbg[2];
  int* nbg_cnt[2];
  int nbg_stride;
  // Per particle: bound on the distance moved since the last full build of the lists
  // (permuted with the particles, into the other buffer).
  float* dacc[2];
  unsigned* nbb[2];  // boundary particles' kept lists, the same form with stride npb
  int* nbb_cnt[2];
  int* inv;          // inverse of the last permutation: new index of old index j
  int* queue;        // rows whose lists a list update rebuilds (Dyn::n_queue of them)
  unsigned* cell_mark;  // per cell: generation of its last mark (listed in marks when first marked)
  int* marks;           // the cells marked in the current generation (Dyn::n_marks, at most RW_MARK_CAP)
  unsigned* near_mark;  // per cell: generation of the last mark in its 27-cell neighbourhood
  unsigned char* near_wall;  // per cell: a contact-wall particle lies in its 27-cell neighbourhood
};

// Distinct cells one list update takes; more marked cells make it a full build.
constexpr int RW_MARK_CAP = 8192;

// Interaction block size; capacity of a kept candidate list (entries per particle).
constexpr int IX_THREADS = 128, IX_CAP = 96;
// The walk launch takes 64 or 128 (default) threads per block (RW_OPT_WALK_THREADS); a
// launch bound of 256 made the same code 14% slower.
constexpr int IX_WALK_MAX_THREADS = 128;

template <class T> RWD V3<T> ld3(const V4<T>* p, int i) { V4<T> v = p[i]; return {v.x, v.y, v.z}; }
template <class T> RWD S6<T> ld6(const V4<T>* a, const V2<T>* b, int i) {
  V4<T> x = a[i];
  V2<T> y = b[i];
  return {x.x, x.y, x.z, x.w, y.x, y.y};
}
template <class T> RWD void st6(V4<T>* a, V2<T>* b, int i, S6<T> s) {
  a[i] = V4<T>{s.xx, s.yy, s.zz, s.xy};
  b[i] = V2<T>{s.xz, s.yz};
}
template <class T> RWD bool in_grid(const Params<T>& P, I3 c) {
  return c.x >= 0 && c.y >= 0 && c.z >= 0 && c.x < P.cell_num[0] && c.y < P.cell_num[1] && c.z < P.cell_num[2];
}
template <class T> RWD int key_of(const Params<T>& P, I3 c) {
  return c.x * P.cell_num[1] * P.cell_num[2] + c.y * P.cell_num[2] + c.z;
}
RWD I3 off_of(int oc) { return {oc % 3 - 1, (oc / 3) % 3 - 1, oc / 9 - 1}; }

// Entry of a kept list: particle index in the low 26 bits, the digits dx, dy, dz (0..2) of
// its cell's offset plus one in two bits each above them.  One shift and a mask per digit
// give the offset (a digit of an offset number takes a multiply and two more operations),
// which the walk pays per entry; lists are kept for np < 2^26 (lists_fit).
constexpr unsigned kEntIdx = 0x3ffffffu;
RWD unsigned list_entry(int j, int oc) {
  return (unsigned)j | ((unsigned)(oc % 3) << 26) | ((unsigned)((oc / 3) % 3) << 28) | ((unsigned)(oc / 9) << 30);
}
RWD I3 entry_off(unsigned e) { return {(int)(e >> 26 & 3u) - 1, (int)(e >> 28 & 3u) - 1, (int)(e >> 30) - 1}; }
// Quad q of the list of column t (lists of `stride` columns).
RWD size_t quad_at(int q, size_t stride, int t) { return ((size_t)q * stride + t) * 4; }
RWD uint4 load_quad(const unsigned* __restrict__ lists, int q, size_t stride, int t) {
  return __ldcs(reinterpret_cast<const uint4*>(lists + quad_at(q, stride, t)));
}
// Entries of one list written in order, a quad at a time.
struct QuadWriter {
  unsigned* lists;
  size_t stride;
  int t, cnt = 0;
  unsigned a = 0, b = 0, c = 0;
  RWD void push(unsigned e, int cap) {
    const int k = cnt & 3;
    if (k == 3) {
      if (cnt < cap) __stcs(reinterpret_cast<uint4*>(lists + quad_at(cnt >> 2, stride, t)), uint4{a, b, c, e});
    } else {
      if (k == 0) a = e;
      else if (k == 1) b = e;
      else c = e;
    }
    ++cnt;
  }
  // the last quad, filled up with `own` (any valid entry)
  RWD void finish(unsigned own, int cap) {
    const int k = cnt & 3;
    if (k && cnt <= cap)
      __stcs(reinterpret_cast<uint4*>(lists + quad_at(cnt >> 2, stride, t)),
             uint4{a, k > 1 ? b : own, k > 2 ? c : own, own});
  }
};
constexpr int kOwnCell = 13;  // offset number of a particle's own cell

RWD float mul_rn(float a, float b) { return __fmul_rn(a, b); }
RWD float rmul(float a, float b) { return __fmul_rn(a, b); }
RWD double rmul(double a, double b) { return __dmul_rn(a, b); }
RWD double mul_rn(double a, double b) { return __dmul_rn(a, b); }
RWD float add_rn(float a, float b) { return __fadd_rn(a, b); }
RWD double add_rn(double a, double b) { return __dadd_rn(a, b); }

// Neighbour record of particle i (boundary: mass = V0 rho; material: idmassidx.y),
// with the reference's per-pair expressions (src/particle_interaction.cu:44-49,71).
template <class T> RWD void write_rec(const Params<T>& P, Rec<T>* rec, int i, V4<T> pos, V4<T> vr, S6<T> s, T mass,
                                      bool contact) {
  const T rho = vr.w;
  const S6<T> sor = s / rmul(rho, rho);
  const T vol = mass / rho;
  Rec<T> r;
  r.p = V4<T>{pos.x, pos.y, pos.z, T(0)};
  r.vr = vr;
  r.a = V4<T>{mass, contact ? -vol : vol, sor.xx, sor.yy};
  r.b = V4<T>{sor.zz, sor.xy, sor.xz, sor.yz};
  if constexpr (sizeof(T) == 4) {  // two 256-bit stores (sm_100)
    float* q = reinterpret_cast<float*>(rec + i);
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(q), "f"(r.p.x), "f"(r.p.y), "f"(r.p.z),
                 "f"(r.p.w), "f"(r.vr.x), "f"(r.vr.y), "f"(r.vr.z), "f"(r.vr.w)
                 : "memory");
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(q + 8), "f"(r.a.x), "f"(r.a.y),
                 "f"(r.a.z), "f"(r.a.w), "f"(r.b.x), "f"(r.b.y), "f"(r.b.z), "f"(r.b.w)
                 : "memory");
  } else {
    rec[i] = r;
  }
}

// The neighbour-side values one pair term needs.
template <class T> struct NbVals {
  V4<T> p, vr, a, b;
};
template <class T> RWD NbVals<T> load_nb(const Rec<T>* __restrict__ rec, int j) {
  NbVals<T> v;
  v.p = rec[j].p;
  v.vr = rec[j].vr;
  v.a = rec[j].a;
  v.b = rec[j].b;
  return v;
}
// Float records: two 256-bit loads (sm_100) instead of four 128-bit ones.  Half the load
// instructions and L1 requests per neighbour; the walk kernel's L1 request rate is what
// bounds it.  Records are 64 bytes from a 256-byte aligned cudaMalloc base.
static_assert(sizeof(Rec<float>) == 64, "float records are one 64-byte line");
template <> RWD NbVals<float> load_nb<float>(const Rec<float>* __restrict__ rec, int j) {
  NbVals<float> v;
  const float* q = reinterpret_cast<const float*>(rec + j);
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(v.p.x), "=f"(v.p.y), "=f"(v.p.z), "=f"(v.p.w), "=f"(v.vr.x), "=f"(v.vr.y), "=f"(v.vr.z), "=f"(v.vr.w)
      : "l"(q));
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(v.a.x), "=f"(v.a.y), "=f"(v.a.z), "=f"(v.a.w), "=f"(v.b.x), "=f"(v.b.y), "=f"(v.b.z), "=f"(v.b.w)
      : "l"(q + 8));
  return v;
}

// ---------------------------------------------------------------------------------
// Case ingest: the caller's arrays (array of structures, double) -> the device layout.
// ---------------------------------------------------------------------------------
struct RawCase {
  const int4* codes;
  const double* pospres;
  const double* velrhop;
  const double* idmassidx;
  const double* stress;
  const double* strain;
  const double* normal;
};

// One particle of LoadParticles' values with the absolute -> in-cell split of
// PositionFromAbsolute2Relative (src/loquat_grid.cu:253-271): cell = trunc(x * (0.5/h)),
// the product rounded on its own, in-cell position = x - cell * 2h with one rounding, as
// the reference's kernel computes them.
template <class T> __global__ void k_ingest(const Params<T> P, DevState<T> S, RawCase R, T half_ih) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= (size_t)P.np) return;
  S.codes[0][i] = R.codes[i];
  const double* a = R.pospres + 4 * i;
  const V4<T> pa{(T)a[0], (T)a[1], (T)a[2], (T)a[3]};
  S.pos_ori[0][i] = pa;
  const int cx = (int)rmul(pa.x, half_ih), cy = (int)rmul(pa.y, half_ih), cz = (int)rmul(pa.z, half_ih);
  S.cellpos[0][i] = int4{cx, cy, cz, 0};
  // x - c 2h as one fused multiply-add: the reference's kernel (cuPositionFromAbsolute2Relative,
  // src/loquat_grid.cu:253-261) is compiled with contraction, which fuses that product
  // into the subtraction
  S.pos[0][i] = V4<T>{f_fma(-(T)cx, P.two_h, pa.x), f_fma(-(T)cy, P.two_h, pa.y), f_fma(-(T)cz, P.two_h, pa.z), pa.w};
  a = R.velrhop + 4 * i;
  S.vel[0][i] = V4<T>{(T)a[0], (T)a[1], (T)a[2], (T)a[3]};
  a = R.idmassidx + 4 * i;
  S.idm[0][i] = V4<T>{(T)a[0], (T)a[1], (T)i, (T)a[3]};
  a = R.stress + 6 * i;
  S.str_a[0][i] = V4<T>{(T)a[0], (T)a[1], (T)a[2], (T)a[3]};
  S.str_b[0][i] = V2<T>{(T)a[4], (T)a[5]};
  a = R.strain + 6 * i;
  S.stn_a[0][i] = V4<T>{(T)a[0], (T)a[1], (T)a[2], (T)a[3]};
  S.stn_b[0][i] = V2<T>{(T)a[4], (T)a[5]};
  if (i < (size_t)P.npb) {
    a = R.normal + 4 * i;
    S.normal[0][i] = V4<T>{(T)a[0], (T)a[1], (T)a[2], (T)a[3]};
  }
}

// ---------------------------------------------------------------------------------
// Cell list: keys, stable radix sort, ranges, gather-permute
// (src/loquat_grid.cu:71-261, src/loquat.cu:254-287).
// ---------------------------------------------------------------------------------

// cuGetParticleCellIndex (src/loquat_grid.cu:71-95).  A live particle whose cell is
// outside the grid would make the reference write out of bounds; here its key is
// clamped into the grid and RW_DERR_CELL_RANGE is raised.
template <class T> __global__ void k_keys(const Params<T> P, DevState<T> S, Dyn<T>* dyn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) dyn->need_sort = 0;
  if (i >= P.np || !dyn->cells_dirty) return;  // no cell changed: keys, order and ranges stand
  const int c = dyn->cur_main;
  int4 cp = S.cellpos[c][i];
  int key;
  if (cp.w == P.ncell_delete_m) {
    key = P.ncell_delete_m;
  } else {
    I3 cc{cp.x, cp.y, cp.z};
    if (!in_grid(P, cc)) {
      atomicOr(&dyn->err, 1u);
      cc.x = min(max(cc.x, 0), P.cell_num[0] - 1);
      cc.y = min(max(cc.y, 0), P.cell_num[1] - 1);
      cc.z = min(max(cc.z, 0), P.cell_num[2] - 1);
    }
    key = key_of(P, cc);
    if (!(S.idm[c][i].x < T(RW_MATERIAL_NUMBER))) key += P.ncell_material;
    S.cellpos[c][i].w = key;
  }
  S.keys[i] = key;
  S.vals[i] = i;
}

static __global__ void k_check_sorted(const int* keys, int n, int* need_sort, const int* dirty = nullptr) {
  if (dirty && !*dirty) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const bool out_of_order = i < n && keys[i - 1] > keys[i];
  // one store per warp that found a key out of order: in an unsorted array every thread
  // would otherwise store to the same word (measured 50 us instead of 6 us at 0.96M)
  if (__any_sync(0xffffffffu, out_of_order) && (threadIdx.x & 31) == 0) *need_sort = 1;
}

// Clears n words when the cells changed since the last search.
static __global__ void k_clear_if(unsigned* p, size_t n, const int* dirty) {
  if (!*dirty) return;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) p[k] = 0u;
}

// Stable LSD radix sort of cell keys with their permutation: per digit an upsweep (digit
// counts per tile), a scan (over the tiles, per digit) and a downsweep (stable ranks in the
// tile, scatter).  All three return immediately when the keys are already in order (the
// permutation is then the identity, exactly what a stable sort of sorted keys returns).
//
// What bounds it is latency: launches, and in the downsweep the block's barriers.  A warp
// takes a run of the tile's keys and ranks them against counts of its own, so a tile needs
// three barriers whatever its size (four per 256 keys with counts shared by the block), and
// digits are as wide as the tables allow: two passes for the grids of walls up to two million
// particles instead of three of eight bits.  1,000,003 keys below 2 10^6 (three passes
// either way): 109 us a sort, 62 now; a wall's sorted section at 674,786 particles: 300 us with
// the old sort, 270 now.
constexpr int RS_THREADS = 256, RS_WARPS = RS_THREADS / 32, RS_MAX_BITS = 11;
struct SortPlan {
  int passes, bits, items, tiles;  // digits of `bits` bits; tiles of RS_THREADS * items keys
  int bins() const { return 1 << bits; }
  int tile() const { return RS_THREADS * items; }
  size_t hist() const { return (size_t)bins() * tiles; }  // counts per tile and digit
};
// Keys of key_bits bits, counts limited to max_hist.  Items per thread: large inputs take
// larger tiles (fewer counts), small ones spread over the SMs.
static inline SortPlan sort_plan(long n, int key_bits, size_t max_hist, int max_bits = RS_MAX_BITS) {
  for (int passes = (key_bits + max_bits - 1) / max_bits;; ++passes) {
    SortPlan p;
    p.passes = passes;
    p.bits = (key_bits + passes - 1) / passes;
    for (p.items = n > (1 << 19) ? 16 : n > (1 << 17) ? 8 : 4; p.items <= 16; p.items *= 2) {
      p.tiles = (int)((n + p.tile() - 1) / p.tile());
      if (p.hist() <= max_hist) return p;
    }
    if (p.bits <= 1) return p;
  }
}

template <int Items>
static __global__ void __launch_bounds__(RS_THREADS) k_rs_upsweep(const int* __restrict__ keys, int n, int shift, int bins,
                                                                  int* __restrict__ hist, const int* need) {
  if (need && !*need) return;
  extern __shared__ int h[];
  const int t = threadIdx.x;
  for (int d = t; d < bins; d += RS_THREADS) h[d] = 0;
  __syncthreads();
  const int base = blockIdx.x * RS_THREADS * Items;
  int key[Items];
#pragma unroll
  for (int k = 0; k < Items; ++k) {
    const int idx = base + k * RS_THREADS + t;
    key[k] = idx < n ? keys[idx] : -1;
  }
#pragma unroll
  for (int k = 0; k < Items; ++k)
    if (base + k * RS_THREADS + t < n) atomicAdd(&h[(key[k] >> shift) & (bins - 1)], 1);
  __syncthreads();
  for (int d = t; d < bins; d += RS_THREADS) hist[(size_t)blockIdx.x * bins + d] = h[d];
}

static __device__ __forceinline__ int block_excl_scan256(int v, int* total) {
  __shared__ int ws[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = lane < 8 ? ws[lane] : 0;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < 8) ws[lane] = s;
  }
  __syncthreads();
  int incl = x + (w > 0 ? ws[w - 1] : 0);
  if (total) *total = ws[7];
  __syncthreads();
  return incl - v;
}

// Exclusive prefix of every digit's counts over the tiles, and the digits' totals: a block
// takes 32 digits (a warp reads them side by side), its warps consecutive runs of tiles.
constexpr int RS_SCAN_WARPS = 32, RS_SCAN_HELD = 16;
static __global__ void __launch_bounds__(RS_SCAN_WARPS * 32) k_rs_scan(int* __restrict__ hist, int tiles, int bins,
                                                                      int* __restrict__ dtot, const int* need) {
  if (need && !*need) return;
  __shared__ int part[RS_SCAN_WARPS][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = blockIdx.x * 32 + lane;
  const int b = (int)((long)tiles * w / RS_SCAN_WARPS), e = (int)((long)tiles * (w + 1) / RS_SCAN_WARPS);
  int held[RS_SCAN_HELD];  // the first counts stay in registers for the second round
  int s = 0;
#pragma unroll
  for (int k = 0; k < RS_SCAN_HELD; ++k) held[k] = d < bins && b + k < e ? hist[(size_t)(b + k) * bins + d] : 0;
#pragma unroll
  for (int k = 0; k < RS_SCAN_HELD; ++k) s += held[k];
  if (d < bins) {
#pragma unroll 8
    for (int k = b + RS_SCAN_HELD; k < e; ++k) s += hist[(size_t)k * bins + d];
  }
  part[w][lane] = s;
  __syncthreads();
  {  // warp w: prefix of digit w of the 32 over the warps' sums
    const int v = part[lane][w];
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    part[lane][w] = x - v;
    if (lane == 31 && blockIdx.x * 32 + w < bins) dtot[blockIdx.x * 32 + w] = x;
  }
  __syncthreads();
  if (d < bins) {
    int off = part[w][lane];
#pragma unroll
    for (int k = 0; k < RS_SCAN_HELD; ++k)
      if (b + k < e) {
        hist[(size_t)(b + k) * bins + d] = off;
        off += held[k];
      }
#pragma unroll 8
    for (int k = b + RS_SCAN_HELD; k < e; ++k) {
      const int v = hist[(size_t)k * bins + d];
      hist[(size_t)k * bins + d] = off;
      off += v;
    }
  }
}

// Shared memory of a downsweep block: the tile's keys and values in order, each digit's first
// position in the output less that in the tile, and each warp's counts.
static inline size_t rs_down_smem(int bins, int tile) {
  return (size_t)tile * sizeof(int2) + (size_t)bins * (sizeof(int) + RS_WARPS * sizeof(unsigned short));
}
template <int Items>
static __global__ void __launch_bounds__(RS_THREADS) k_rs_downsweep(const int* __restrict__ kin, const int* __restrict__ vin,
                                                                    int* __restrict__ kout, int* __restrict__ vout, int n,
                                                                    int shift, int bins, const int* __restrict__ hist,
                                                                    const int* __restrict__ dtot, const int* need) {
  if (need && !*need) return;
  extern __shared__ int2 kv[];
  int* base = reinterpret_cast<int*>(kv + RS_THREADS * Items);
  unsigned short* wcnt = reinterpret_cast<unsigned short*>(base + bins);  // [warp][digit]
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int tile0 = blockIdx.x * RS_THREADS * Items, first = tile0 + w * 32 * Items;
  int key[Items], val[Items];
#pragma unroll
  for (int k = 0; k < Items; ++k) {
    const int idx = first + k * 32 + lane;
    key[k] = idx < n ? kin[idx] : 0;
    val[k] = idx < n ? (vin ? vin[idx] : idx) : 0;
  }
  const int per = (bins + RS_THREADS - 1) / RS_THREADS, d0 = min(t * per, bins), d1 = min(d0 + per, bins);
  int out = 0;  // output position of this thread's first digit: the smaller digits' totals
  for (int d = d0; d < d1; ++d) out += dtot[d];
  for (int d = t; d < bins * RS_WARPS / 2; d += RS_THREADS) reinterpret_cast<unsigned*>(wcnt)[d] = 0u;
  out = block_excl_scan256(out, nullptr);
  // Ranks within the warp's run, in order.  The lanes of equal digit come from one vote per
  // bit, all keys' votes side by side (a match over 32 different digits takes them one after
  // the other: 25 us a downsweep of a million keys, 19 with votes).
  unsigned short* mine = wcnt + (size_t)w * bins;
  unsigned peers[Items];
  int rank[Items];
#pragma unroll
  for (int k = 0; k < Items; ++k) peers[k] = __ballot_sync(0xffffffffu, first + k * 32 + lane < n);
  for (int b = 1; b < bins; b <<= 1) {
#pragma unroll
    for (int k = 0; k < Items; ++k) {
      const bool one = key[k] >> shift & b;
      const unsigned v = __ballot_sync(0xffffffffu, one);
      peers[k] &= one ? v : ~v;
    }
  }
#pragma unroll
  for (int k = 0; k < Items; ++k) {
    const bool valid = first + k * 32 + lane < n;
    const int d = (key[k] >> shift) & (bins - 1);
    const int before = valid ? mine[d] : 0;
    rank[k] = before + __popc(peers[k] & ((1u << lane) - 1u));
    __syncwarp();
    if (valid && lane == __ffs(peers[k]) - 1) mine[d] = (unsigned short)(before + __popc(peers[k]));
    __syncwarp();
  }
  __syncthreads();
  // every digit's first place in the tile, the earlier warps' counts on top of it
  int in_tile = 0;
  for (int d = d0; d < d1; ++d)
#pragma unroll
    for (int q = 0; q < RS_WARPS; ++q) in_tile += wcnt[(size_t)q * bins + d];
  in_tile = block_excl_scan256(in_tile, nullptr);
  for (int d = d0; d < d1; ++d) {
    base[d] = out + hist[(size_t)blockIdx.x * bins + d] - in_tile;
    out += dtot[d];
#pragma unroll
    for (int q = 0; q < RS_WARPS; ++q) {
      const int v = wcnt[(size_t)q * bins + d];
      wcnt[(size_t)q * bins + d] = (unsigned short)in_tile;
      in_tile += v;
    }
  }
  __syncthreads();
  // The tile in order first, so that a digit's run leaves in whole sectors: single scattered
  // words cost a 32-byte sector each (19 us a downsweep of a million random keys, 11 staged).
#pragma unroll
  for (int k = 0; k < Items; ++k) {
    if (first + k * 32 + lane >= n) continue;
    const int d = (key[k] >> shift) & (bins - 1);
    kv[mine[d] + rank[k]] = int2{key[k], val[k]};
  }
  __syncthreads();
  const int count = min(RS_THREADS * Items, n - tile0);
#pragma unroll
  for (int k = 0; k < Items; ++k) {
    const int at = k * RS_THREADS + t;
    if (at >= count) continue;
    const int2 x = kv[at];
    const int pos = base[(x.x >> shift) & (bins - 1)] + at;
    if (pos >= 0 && pos < n) {  // always true for consistent counts; guards the scatter
      kout[pos] = x.x;
      vout[pos] = x.y;
    }
  }
}

// One pass of the sort on stream st.
template <int Items>
static void rs_pass_items(const SortPlan& p, const int* kin, const int* vin, int* kout, int* vout, int n, int pass, int* hist,
                          int* dtot, const int* need, cudaStream_t st) {
  const int shift = pass * p.bits, bins = p.bins();
  k_rs_upsweep<Items><<<p.tiles, RS_THREADS, bins * sizeof(int), st>>>(kin, n, shift, bins, hist, need);
  k_rs_scan<<<(bins + 31) / 32, RS_SCAN_WARPS * 32, 0, st>>>(hist, p.tiles, bins, dtot, need);
  k_rs_downsweep<Items><<<p.tiles, RS_THREADS, rs_down_smem(bins, p.tile()), st>>>(kin, vin, kout, vout, n, shift, bins, hist, dtot, need);
}
static inline void rs_pass(const SortPlan& p, const int* kin, const int* vin, int* kout, int* vout, int n, int pass, int* hist,
                           int* dtot, const int* need, cudaStream_t st) {
  if (p.items == 4) rs_pass_items<4>(p, kin, vin, kout, vout, n, pass, hist, dtot, need, st);
  else if (p.items == 8) rs_pass_items<8>(p, kin, vin, kout, vout, n, pass, hist, dtot, need, st);
  else rs_pass_items<16>(p, kin, vin, kout, vout, n, pass, hist, dtot, need, st);
}

// cuFindBegEndInCell (src/loquat_grid.cu:116-144): [beg, end) of every occupied cell.
template <class T> __global__ void k_ranges(const Params<T> P, DevState<T> S, const Dyn<T>* dyn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.np || !dyn->cells_dirty) return;
  const int* K = dyn->need_sort ? S.skeys : S.keys;
  const int k = K[i];
  int* r = reinterpret_cast<int*>(S.range);
  if (i == 0 || K[i - 1] != k) r[2 * k] = i;
  if (i == P.np - 1 || K[i + 1] != k) r[2 * k + 1] = i + 1;
}

// Deleted-particle accounting (src/loquat_grid.cu:164-190), on the device.
template <class T> __global__ void k_count(const Params<T> P, DevState<T> S, Dyn<T>* dyn) {
  if (!dyn->cells_dirty) return;
  int2 d = S.range[P.ncell_delete_m];
  int cnt = d.y - d.x;
  if (cnt > 0) {
    int now = cnt - dyn->np_delete_m;
    if (now != 0) {
      dyn->npm -= now;
      dyn->np_delete_m += now;
    }
  }
  if (P.npb + dyn->npm + dyn->np_delete_m != P.np) atomicOr(&dyn->err, 2u);
}

// SortArraysPrimary (section 0) / SortArraysAll (section 1), src/loquat.cu:254-287,
// as one gather into the other ping-pong buffer.  Stress/strain beyond npb+npm are
// not part of the reference's sorted range; they keep their slot values.
template <class T> __global__ void k_permute(const Params<T> P, DevState<T> S, const Dyn<T>* dyn, int section,
                                             int compat_contact) {
  if (!dyn->need_sort) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.np) return;
  int j = S.sperm[i];
  if (j < 0 || j >= P.np) {  // a valid permutation never gets here
    atomicOr(&const_cast<Dyn<T>*>(dyn)->err, 8u);
    j = i;
  }
  const int c = dyn->cur_main, n = c ^ 1;
  S.codes[n][i] = S.codes[c][j];
  S.cellpos[n][i] = S.cellpos[c][j];
  S.pos[n][i] = S.pos[c][j];
  S.pos_ori[n][i] = S.pos_ori[c][j];
  S.vel[n][i] = S.vel[c][j];
  S.idm[n][i] = S.idm[c][j];
  if (P.mixed) {
    S.cmp_p[n][i] = S.cmp_p[c][j];
    S.cmp_v[n][i] = S.cmp_v[c][j];
  }
  // the lists' displacement bounds move with the particles (k_flip then flips lbuf), and
  // a list update maps the entries through the inverse
  const int lb = dyn->lbuf;
  S.dacc[lb ^ 1][i] = S.dacc[lb][j];
  S.inv[j] = i;
  const int npm = dyn->npm;
  const int nbm = P.npb + npm;
  const bool perm_str = (section == 0) || (npm != 0);
  const int ss = (perm_str && i < nbm) ? j : i;
  S.str_a[n][i] = S.str_a[c][ss];
  S.str_b[n][i] = S.str_b[c][ss];
  S.stn_a[n][i] = S.stn_a[c][ss];
  S.stn_b[n][i] = S.stn_b[c][ss];
  if (section == 0) {
    const int cn = dyn->cur_nrm;
    if (i < P.npb) S.normal[cn ^ 1][i] = S.normal[cn][j];
  } else {
    const int ci = dyn->cur_ini, ni = ci ^ 1;
    S.pos_ini[ni][i] = S.pos_ini[ci][j];
    S.vel_ini[ni][i] = S.vel_ini[ci][j];
    S.stri_a[ni][i] = S.stri_a[ci][ss];
    S.stri_b[ni][i] = S.stri_b[ci][ss];
    S.stni_a[ni][i] = S.stni_a[ci][ss];
    S.stni_b[ni][i] = S.stni_b[ci][ss];
    if (P.mixed) {
      S.cmp_pi[ni][i] = S.cmp_pi[ci][j];
      S.cmp_vi[ni][i] = S.cmp_vi[ci][j];
    }
  }
  (void)compat_contact;
}

// Buffer flip after a permute; in the predictor section also RigidBodyUpdate
// (src/adami_boundary.cu:175-203), which the reference runs right after the sort.
// Plain round-to-nearest products/sums, as the reference's host code computes.
template <class T> __global__ void k_flip(const Params<T> P, Dyn<T>* dyn, int section, int rigid, int lists) {
  if (section >= 0 && dyn->need_sort) {
    dyn->cur_main ^= 1;
    if (section == 0) dyn->cur_nrm ^= 1;
    else dyn->cur_ini ^= 1;
    dyn->n_sorts += 1;
    dyn->lbuf ^= 1;  // k_permute carried the displacement bounds into the other buffer
  }
  // Candidate lists.  An interaction walks the kept lists (mode 1) when nothing was
  // permuted and no particle changed cell since they were built or updated.  When
  // particles changed cell (marked cells) in the step before a predictor section, the
  // lists are updated (mode 2): the lists of particles next to a marked cell are
  // rebuilt, the others carried through the permutation.  Every list is built anew
  // (mode 0) when some particle moved more than the skin allows since the last full
  // build (list_kill, raised by the integrators), after a host write, with too many
  // marked cells, or in the corrector section: lists built there, from mid-step
  // positions, are not kept, and a displacement bound counted from the start of the
  // step does not cover them.  Without kept soil lists (lists = 0: lists off, or the
  // chunked kernel) every section is mode 0 and no list stands.
  if (section >= 0) {
    if (dyn->need_sort || dyn->host_dirty) dyn->rec_stale = 1;  // until the next interaction
    dyn->host_dirty = 0;
    dyn->cells_dirty = 0;  // the search is complete
    int mode = 1;
    if (!lists || !dyn->list_ok || dyn->list_kill || dyn->n_marks > RW_MARK_CAP) mode = 0;
    else if (dyn->need_sort || dyn->n_marks > 0) mode = section == 0 ? 2 : 0;
    dyn->ix_mode = mode;
    dyn->n_reuse += mode == 1;
    dyn->n_updates += mode == 2;
    // the marks are consumed: the update tests this generation, new marks take the next
    dyn->near_gen = dyn->mark_gen;
    dyn->mark_gen += 1;
    dyn->n_marks = 0;
    dyn->n_queue = 0;
    if (mode == 0) {
      dyn->list_ok = 0;
      dyn->list_kill = 0;
      dyn->build_kill = section;
      dyn->n_spill = 0;
    }
  }
  if (!rigid) return;
  const T dt = P.dt;
  const T time = dyn->time_f;
  for (int i = 0; i < P.n_motion; ++i) {
    Table<T>& tb = dyn->tab[i];
    Motion<T>& mv = dyn->mv[i];
    if (tb.is_rotation) {
      for (int j = 0; j < tb.n_rot; ++j) {
        if (time < tb.rotat_time[j]) {
          tb.rotat_vel.x = add_rn(tb.rotat_vel.x, mul_rn(tb.rotat_acc[j].x, dt));
          tb.rotat_vel.y = add_rn(tb.rotat_vel.y, mul_rn(tb.rotat_acc[j].y, dt));
          tb.rotat_vel.z = add_rn(tb.rotat_vel.z, mul_rn(tb.rotat_acc[j].z, dt));
          const T hdt = (T)(0.5 * (double)dt);
          Vec3<T> vel{add_rn(tb.trans_vel[j].x, mul_rn(tb.trans_acc[j].x, hdt)),
                      add_rn(tb.trans_vel[j].y, mul_rn(tb.trans_acc[j].y, hdt)),
                      add_rn(tb.trans_vel[j].z, mul_rn(tb.trans_acc[j].z, hdt))};
          tb.pos_rp.x = add_rn(tb.pos_rp.x, mul_rn(vel.x, dt));
          tb.pos_rp.y = add_rn(tb.pos_rp.y, mul_rn(vel.y, dt));
          tb.pos_rp.z = add_rn(tb.pos_rp.z, mul_rn(vel.z, dt));
          mv.rotat_acc = tb.rotat_acc[j];
          mv.rotat_vel = tb.rotat_vel;
          mv.pos_rp = tb.pos_rp;
          break;
        }
      }
    }
    if (tb.is_translation) {
      for (int j = 0; j < tb.n_trans; ++j) {
        if (time < tb.trans_time[j]) {
          tb.trans_vel[j].x = add_rn(tb.trans_vel[j].x, mul_rn(tb.trans_acc[j].x, dt));
          tb.trans_vel[j].y = add_rn(tb.trans_vel[j].y, mul_rn(tb.trans_acc[j].y, dt));
          tb.trans_vel[j].z = add_rn(tb.trans_vel[j].z, mul_rn(tb.trans_acc[j].z, dt));
          mv.trans_acc = tb.trans_acc[j];
          mv.trans_vel = tb.trans_vel[j];
          break;
        }
      }
    }
  }
}

// Gates of a captured step graph: one-thread kernels that set the condition of the IF
// node holding work that would otherwise launch only to return at once.
// Search: keys, sort, ranges, counts, permutation and contact-wall cells have nothing to
// do when no particle changed cell (what k_keys does then is clear need_sort).
template <class T> __global__ void k_search_gate(Dyn<T>* dyn, cudaGraphConditionalHandle h) {
  const int d = dyn->cells_dirty;
  if (!d) {
    dyn->need_sort = 0;
    dyn->n_search_skipped += 1;
  }
  cudaGraphSetConditional(h, d ? 1u : 0u);
}
// List build: needed when the lists are to be built or updated (modes 0 and 2, lists on).
template <class T>
__global__ void k_build_gate(const Params<T> P, DevState<T> S, Dyn<T>* dyn, cudaGraphConditionalHandle h) {
  const bool run = S.nbg[0] && P.keep_lists && dyn->ix_mode != 1;
  if (!run) dyn->n_build_skipped += 1;
  cudaGraphSetConditional(h, run ? 1u : 0u);
}
// Interaction scan launch: needed with lists off, when some list of the last build
// overflowed, or for deleted slots (their contact state is carried).
template <class T>
__global__ void k_scan_gate(const Params<T> P, DevState<T> S, Dyn<T>* dyn, cudaGraphConditionalHandle h) {
  const bool run = !(S.nbg[0] && P.keep_lists) || dyn->n_spill > 0 || dyn->npm < P.np - P.npb;
  if (!run) {
    dyn->rec_stale = 0;  // what the scan launch does first
    dyn->n_scan_skipped += 1;
  }
  cudaGraphSetConditional(h, run ? 1u : 0u);
}

template <class T> __global__ void k_begin(Dyn<T>* dyn) { dyn->time_f = (T)dyn->time_d; }
template <class T> __global__ void k_end(const Params<T> P, Dyn<T>* dyn) {
  dyn->time_d += (double)P.dt;
  dyn->step += 1;
}

// ---------------------------------------------------------------------------------
// Periodic planes (period-bound cases).  Dist2Plane / AbsDist2Plane
// (src/functions.h:134-139); every operation separately rounded, so the decisions and
// the image coordinates match the oracle bit for bit.
// ---------------------------------------------------------------------------------
template <class T> RWD T plane_dist(const T* pl, const V3<T> a) {
  using F = Fp<true>;
  const T num = F::mad(a.z, pl[2], F::mad(a.y, pl[1], F::mul(a.x, pl[0]))) + pl[3];
  return num / pair_r(pair_r2(pl[0], pl[1], pl[2]));
}

template <class T> RWD V3<T> abs_pos(const V3<T> p, const I3 c, T th) {
  using F = Fp<true>;
  return V3<T>{F::mad((T)c.x, th, p.x), F::mad((T)c.y, th, p.y), F::mad((T)c.z, th, p.z)};
}

// Absolute position pabs moved by one period along the plane pl, as a cell and an
// in-cell position.
template <class T> RWD void period_shift(const Params<T>& P, const V3<T> pabs, const T* pl, T len, I3& cpb,
                                         V3<T>& ppb) {
  using F = Fp<true>;
  const V3<T> pb{F::mad(pl[0], len, pabs.x), F::mad(pl[1], len, pabs.y), F::mad(pl[2], len, pabs.z)};
  const T s = F::mul(T(0.5f), P.i_h);
  cpb = I3{int(F::mul(pb.x, s)), int(F::mul(pb.y, s)), int(F::mul(pb.z, s))};
  ppb = V3<T>{F::msub((T)cpb.x, P.two_h, pb.x), F::msub((T)cpb.y, P.two_h, pb.y), F::msub((T)cpb.z, P.two_h, pb.z)};
}

// Periodic image of a particle within 2h of a periodic plane (the *LoopPeriod helpers:
// src/adami_boundary.cu:73-88, src/field_smoothing.cu:58-72,
// src/particle_interaction.cu:243-257).  The period is |D_left + D_right| in the Adami
// and Shepard loops (abs_len) and the signed sum in the interaction.
template <class T> RWD bool period_image(const Params<T>& P, const I3 celli, const V3<T> pos_i, bool abs_len,
                                         I3& cpb, V3<T>& ppb) {
  const V3<T> pabs = abs_pos(pos_i, celli, P.two_h);
  const bool left = f_abs(plane_dist(P.planeleft, pabs)) < P.two_h;
  const bool right = f_abs(plane_dist(P.planeright, pabs)) < P.two_h;
  if (!left && !right) return false;
  T len = P.planeleft[3] + P.planeright[3];
  if (abs_len) len = f_abs(len);
  period_shift(P, pabs, left ? P.planeleft : P.planeright, len, cpb, ppb);
  return true;
}

// A particle that left through a periodic plane re-enters through the other one
// (cuCheckOutDomainPeriod, src/predictor_corrector.cu:26-40).
template <class T> RWD void period_wrap(const Params<T>& P, int4& cp, V4<T>& ps) {
  const V3<T> pabs = abs_pos(xyz(ps), I3{cp.x, cp.y, cp.z}, P.two_h);
  const bool left = plane_dist(P.planeleft, pabs) < T(0.0);
  const bool right = plane_dist(P.planeright, pabs) < T(0.0);
  if (!left && !right) return;
  I3 c;
  V3<T> pr;
  period_shift(P, pabs, left ? P.planeleft : P.planeright, f_abs(P.planeleft[3] + P.planeright[3]), c, pr);
  cp = int4{c.x, c.y, c.z, cp.w};
  ps = V4<T>{pr.x, pr.y, pr.z, ps.w};
}

// A list update rebuilds the list of a particle in cell c when c lies next to a cell
// marked in the generation being consumed; a cell outside the grid (a wall particle
// moved out of it) always counts as marked.
template <class T> RWD bool near_marked(const Params<T>& P, const DevState<T>& S, const Dyn<T>* dyn, I3 c) {
  return !in_grid(P, c) || S.near_mark[key_of(P, c)] == dyn->near_gen;
}

// A kept list carried through a permutation: the list of old index o (column o of the
// other buffer) becomes the list of new index i, each entry's particle index mapped to
// its new index; the cell offsets and the order stand (a stable sort keeps the order
// inside every cell whose particles all stayed).
RWD void carry_list(const unsigned* __restrict__ src, const int* __restrict__ src_cnt, int o, unsigned* __restrict__ dst,
                    int* __restrict__ dst_cnt, int i, size_t stride, const int* __restrict__ inv) {
  const int cnt = src_cnt[o];
  dst_cnt[i] = cnt;
  const int nq = (cnt + 3) >> 2;
  // two quads at a time, their loads and index lookups issued together (a thread waits
  // for two loads per eight entries, not two per entry)
  auto map = [&](unsigned e) { return (unsigned)inv[e & kEntIdx] | (e & ~kEntIdx); };
  auto put = [&](int q, uint4 v) { __stcs(reinterpret_cast<uint4*>(dst + quad_at(q, stride, i)), v); };
  for (int q = 0; q < nq; q += 2) {
    const bool two = q + 1 < nq;
    uint4 v = load_quad(src, q, stride, o), w = two ? load_quad(src, q + 1, stride, o) : v;
    v = uint4{map(v.x), map(v.y), map(v.z), map(v.w)};
    w = uint4{map(w.x), map(w.y), map(w.z), map(w.w)};
    put(q, v);
    if (two) put(q + 1, w);
  }
}

// ---------------------------------------------------------------------------------
// Eight lanes per particle, for cases too small to fill the GPU with a thread per particle:
// there a launch lasts as long as one thread's chain of list entries (two or three waits per
// entry or pair of them, whatever the number of particles).  Here each lane forms the terms
// of one entry of eight, and then every lane adds up to three of the particle's sums over the
// eight entries in list order, from shared memory: each sum is still one chain of fused
// multiply-adds over the list, so it is the sum one thread forms, bit for bit.
// A row holds one entry's terms as five groups of four; a sum's lane multiplies one scalar of
// the row (at x) with three (at y).
// ---------------------------------------------------------------------------------
constexpr int kLanes = 8, kGroupThreads = 128, kRow = 20;
template <class T> struct GroupRows {
  // two buffers: a row is read while the next round's are written; a warp's four particles
  // lie 8 elements apart in their banks
  V4<T> row[2][kGroupThreads / 32][4][(kLanes * kRow + 8) / 4];
};
// The lane's three sums over the rows of one round; bit k of `on`: entry k counts.
template <class T> RWD void group_add(const V4<T>* rows, int x, int y, unsigned on, T (&acc)[3]) {
  const T* r = reinterpret_cast<const T*>(rows);
#pragma unroll
  for (int k = 0; k < kLanes; ++k) {
    const V4<T> v = *reinterpret_cast<const V4<T>*>(r + k * kRow + y);
    const T f = r[k * kRow + x];
    if (on >> k & 1u) {
      acc[0] = f_fma(f, v.x, acc[0]);
      acc[1] = f_fma(f, v.y, acc[1]);
      acc[2] = f_fma(f, v.z, acc[2]);
    }
  }
}
RWD float from_lane(float v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
RWD double from_lane(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
// Entry e of the list of column t, or an entry of the particle itself past the end.
RWD unsigned group_entry(const unsigned* __restrict__ lists, size_t stride, int t, int e, int cnt, unsigned own) {
  return e < cnt ? __ldcs(lists + quad_at(e >> 2, stride, t) + (e & 3)) : own;
}

// ---------------------------------------------------------------------------------
// Adami boundary (src/adami_boundary.cu:26-158).
// ---------------------------------------------------------------------------------
// End of the Adami kernel for boundary particle i: wall normal, extrapolated velocity and
// stress, neighbour record.
template <class T>
RWD void adami_finish(const Params<T>& P, const DevState<T>& S, const Dyn<T>* dyn, int c, int i, bool contact,
                      const int4& code, const V3<T> pos_i, const I3 celli, const V3<T> n_i, const S6<T>& rs,
                      const V4<T>& rps, const V4<T>& rvr) {
  const T nn = f_sqrt(f_fma(n_i.z, n_i.z, f_fma(n_i.y, n_i.y, rmul(n_i.x, n_i.x))));
  if (nn > T(0)) {
    S.cny[i] = V4<T>{n_i.x / nn, n_i.y / nn, n_i.z / nn, T(0)};
  }
  V4<T> vr_out = S.vel[c][i];
  S6<T> str_out;
  if (rps.w > T(0.0f)) {
    const T kersum = rps.w;
    const V3<T> dr_ref = xyz(rps);
    const V4<T> nrm4 = S.normal[dyn->cur_nrm][i];
    const T fcoef = nrm4.w;
    const V3<T> nrm = xyz(nrm4);
    const V3<T> vel_ref = xyz(rvr) / kersum;
    const V3<T> vel_ref_n = nrm * dot(nrm, vel_ref);
    const V3<T> vel_ref_t = vel_ref - vel_ref_n;
    V3<T> vel_rb{T(0.0f), T(0.0f), T(0.0f)};
    if (code.y == 1) {
      const Motion<T>& mv = dyn->mv[code.w];
      vel_rb = V3<T>{mv.trans_vel.x, mv.trans_vel.y, mv.trans_vel.z};
      if (mv.is_rotat) {
        V3<T> pabs = pos_i + mulI(celli, T(2.0f) * P.h);
        V3<T> rp{mv.pos_rp.x, mv.pos_rp.y, mv.pos_rp.z};
        V3<T> w{mv.rotat_vel.x, mv.rotat_vel.y, mv.rotat_vel.z};
        vel_rb = vel_rb + cross(w, pabs - rp);
      }
    }
    const V3<T> vel_rb_n = nrm * dot(nrm, vel_rb);
    const V3<T> vel_rb_t = vel_rb - vel_rb_n;
    const V3<T> vel_ext_n = vel_rb_n * T(2.0f) - vel_ref_n;
    const V3<T> vel_ext_t = fcoef == T(-1.0f) ? vel_rb_t * T(2.0f) - vel_ref_t : vel_ref_t;
    const V3<T> vel_ext = vel_ext_n + vel_ext_t;
    const T rho = rvr.w / kersum;
    vr_out = v4(vel_ext, rho);
    if (contact) {
      vr_out = v4(vel_rb, rho);
      S.cvz[i] = V4<T>{vel_ext.x, vel_ext.y, vel_ext.z, T(0)};
    }
    const S6<T> str_ref = rs / kersum;
    const V3<T> g{P.gravity[0], P.gravity[1], P.gravity[2]};
    str_out = subdiag(str_ref, (g * dr_ref) / kersum);
    S.vel[c][i] = vr_out;
  } else {
    str_out = zero6<T>();
  }
  st6(S.str_a[c], S.str_b[c], i, str_out);
  write_rec(P, S.rec, i, S.pos[c][i], vr_out, str_out, P.vol_def * vr_out.w, contact);
}

// Sums of one boundary particle.  The products are explicit fused multiply-adds, so the list
// walks and the scan add alike.
template <class T> struct AdamiSums {
  S6<T> rs;        // stress
  V4<T> rps, rvr;  // distance and kernel sum; velocity and density
  V3<T> n_i;       // wall normal
  RWD void add_normal(const Params<T>& P, const V3<T> dr, T q) {
    const V3<T> g = dr * kernel_f(P.kgrad, q);
    n_i = V3<T>{f_fma(-g.x, P.vol_def, n_i.x), f_fma(-g.y, P.vol_def, n_i.y), f_fma(-g.z, P.vol_def, n_i.z)};
  }
  RWD void add_material(const V3<T> dr, T ker, T kv, const V4<T>& v, T m, const S6<T>& s) {
    rs = S6<T>{f_fma(s.xx, kv, rs.xx), f_fma(s.yy, kv, rs.yy), f_fma(s.zz, kv, rs.zz),
               f_fma(s.xy, kv, rs.xy), f_fma(s.xz, kv, rs.xz), f_fma(s.yz, kv, rs.yz)};
    const T km = ker * m;
    rps = V4<T>{f_fma(dr.x, km, rps.x), f_fma(dr.y, km, rps.y), f_fma(dr.z, km, rps.z), add_rn(rps.w, kv)};
    rvr = V4<T>{f_fma(v.x, kv, rvr.x), f_fma(v.y, kv, rvr.y), f_fma(v.z, kv, rvr.z), f_fma(v.w, kv, rvr.w)};
  }
};
// Boundary particle i's neighbours in the 27 cells around cc, in the reference's order:
// boundary ones (contact walls only) feed the wall normal, material ones the extrapolation
// sums.  With `keep`, the candidates within the list radius are recorded (same order).
template <class T>
RWD void adami_scan(const Params<T>& P, const DevState<T>& S, int c, const I3 cc, const V3<T> pp, bool contact,
                    AdamiSums<T>& A, QuadWriter* keep) {
  const V4<T>* __restrict__ pos = S.pos[c];
  for (int oc = 0; oc < 27; ++oc) {
    const I3 off = off_of(oc);
    const I3 cj{cc.x + off.x, cc.y + off.y, cc.z + off.z};
    if (!in_grid(P, cj)) continue;
    const int k = key_of(P, cj);
    const V3<T> o = mulI(off, P.two_h);
    for (int layer = contact ? 0 : 1; layer < 2; ++layer) {
      const int2 rg = S.range[layer ? k + P.ncell_material : k];
      for (int j = rg.x; j < rg.y; ++j) {
        V3<T> dr = pp - ld3(pos, j);
        dr = dr - o;
        const T r2 = pair_r2(dr.x, dr.y, dr.z);
        if (keep && r2 < P.r2_list) keep->push(list_entry(j, oc), IX_CAP);
        if (!(r2 < P.r2_prefilter)) continue;  // conservative: q >= 2 beyond it
        const T q = pair_r(r2) * P.i_h;
        if (!(q < T(2.0f))) continue;
        if (j < P.npb) {
          A.add_normal(P, dr, q);
        } else {
          const T ker = kernel_w(P.knorm, q);
          const V4<T> vj = S.vel[c][j];
          const T mj = S.idm[c][j].y;
          A.add_material(dr, ker, rmul(ker, mj / vj.w), vj, mj, ld6(S.str_a[c], S.str_b[c], j));
        }
      }
    }
  }
}

template <class T> __global__ void __launch_bounds__(128) k_adami(const Params<T> P, DevState<T> S, const Dyn<T>* dyn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.npb) return;
  if (dyn->ix_mode == 0) S.dacc[dyn->lbuf][i] = 0.0f;  // candidate lists are rebuilt from these positions
  if (dyn->npm == 0) return;
  const int c = dyn->cur_main;
  const V4<T>* __restrict__ pos = S.pos[c];
  const V4<T>* __restrict__ vel = S.vel[c];
  const V4<T>* __restrict__ idm = S.idm[c];
  const V4<T>* __restrict__ sa = S.str_a[c];
  const V2<T>* __restrict__ sb = S.str_b[c];
  const V3<T> pos_i = ld3(pos, i);
  const int4 cp = S.cellpos[c][i];
  const I3 celli{cp.x, cp.y, cp.z};
  const int4 code = S.codes[c][i];
  const bool contact = code.x >= 10;
  AdamiSums<T> A{zero6<T>(), V4<T>{T(0), T(0), T(0), T(0)}, V4<T>{T(0), T(0), T(0), T(0)}, V3<T>{T(0), T(0), T(0)}};
  const T th = P.two_h;
  const int lb = dyn->lbuf;
  unsigned* __restrict__ nbb = S.nbb[lb];
  const bool keep = S.nbb[0] && P.keep_lists;
  const int mode = keep ? dyn->ix_mode : 0;
  // In a list update (mode 2) the lists next to a marked cell were rebuilt and the
  // others carried through this section's permutation, if any, before this kernel
  // (k_build_lists, k_rebuild_lists); only a full build (mode 0) keeps them here.
  const bool rebuild = mode == 0;
  const int kept = (mode != 0 && !rebuild) ? S.nbb_cnt[lb][i] : -1;
  if (kept >= 0) {
    // Walk the kept list four entries at a time, each batch's neighbour data loaded
    // together and the next batch's entries loaded while it is in flight: a thread next
    // to the soil waits for about one load per four entries instead of a chain of loads
    // per entry.
    constexpr unsigned kNone = kEntIdx;  // index of no particle (np < 2^26)
    auto entries = [&](int e0, unsigned* ent) {
      uint4 q{kNone, kNone, kNone, kNone};
      if (e0 < kept) q = load_quad(nbb, e0 >> 2, (size_t)P.npb, i);
      ent[0] = q.x;
      ent[1] = e0 + 1 < kept ? q.y : kNone;
      ent[2] = e0 + 2 < kept ? q.z : kNone;
      ent[3] = e0 + 3 < kept ? q.w : kNone;
    };
    unsigned ent[4], nxt[4];
    entries(0, ent);
    for (int e0 = 0; e0 < kept; e0 += 4) {
      V4<T> pj[4], vj[4];
      T mj[4];
      S6<T> sj[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // no particle: the boundary particle itself, its term not added below.  Only the
        // position of a boundary neighbour counts; velocity and stress of boundary rows are
        // written by this launch, so those lanes read the first soil row instead
        const int j = (ent[k] & kNone) == kNone ? i : (int)(ent[k] & kNone), m = max(j, P.npb);
        pj[k] = pos[j];
        vj[k] = vel[m];
        mj[k] = idm[m].y;
        sj[k] = ld6(sa, sb, m);
      }
      entries(e0 + 4, nxt);
      // The four kernels and volumes are formed side by side without a branch (square
      // roots, divisions and the kernel's double products are long chains), then the sums
      // take the entries in order (65 -> 60 us a launch on the 1.92M wall, 38 -> 36 at 335k).
      V3<T> dr[4];
      T q[4], ker[4], kv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        dr[k] = pos_i - V3<T>{pj[k].x, pj[k].y, pj[k].z};
        dr[k] = dr[k] - mulI(entry_off(ent[k]), th);
        const T r2 = pair_r2(dr[k].x, dr[k].y, dr[k].z);
        q[k] = pair_r(r2) * P.i_h;
        if (!(r2 < P.r2_prefilter) || (ent[k] & kNone) == kNone) q[k] = T(2.0f);
        ker[k] = kernel_w(P.knorm, q[k]);
        kv[k] = rmul(ker[k], mj[k] / vj[k].w);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!(q[k] < T(2.0f))) continue;
        if ((int)(ent[k] & kNone) < P.npb) A.add_normal(P, dr[k], q[k]);
        else A.add_material(dr[k], ker[k], kv[k], vj[k], mj[k], sj[k]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) ent[k] = nxt[k];
    }
  } else {
    QuadWriter out{nbb, (size_t)P.npb, i};
    adami_scan<T>(P, S, c, celli, pos_i, contact, A, rebuild && keep ? &out : nullptr);
    if (rebuild && keep) {
      out.finish(list_entry(i, kOwnCell), IX_CAP);
      S.nbb_cnt[lb][i] = out.cnt <= IX_CAP ? out.cnt : -1;
    }
  }
  if (P.periodbound) {
    I3 cpb;
    V3<T> ppb;
    if (period_image(P, celli, pos_i, true, cpb, ppb)) adami_scan<T>(P, S, c, cpb, ppb, contact, A, nullptr);
  }
  adami_finish(P, S, dyn, c, i, contact, code, pos_i, celli, A.n_i, A.rs, A.rps, A.rvr);
}

// The same with eight lanes per boundary particle (small cases, lists kept): the lanes form
// the terms of eight list entries, then lanes 0..5 add the stress, the distance, the velocity,
// the density with the kernel sum, and the normal.  Lists that overflowed are scanned by one
// lane.  56k-particle wall (28k boundary): 31 -> 22 us a launch, column of 693: 15 -> 12.
template <class T>
__global__ void __launch_bounds__(kGroupThreads) k_adami_group(const Params<T> P, DevState<T> S, const Dyn<T>* dyn) {
  __shared__ GroupRows<T> sm;
  const int lane = threadIdx.x & 31, l = lane & (kLanes - 1), g = lane / kLanes, warp = threadIdx.x >> 5;
  const int row = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  const bool live = row < P.npb;
  const int i = live ? row : P.npb - 1;
  const int mode = dyn->ix_mode, lb = dyn->lbuf, c = dyn->cur_main;
  if (live && l == 0 && mode == 0) S.dacc[lb][i] = 0.0f;  // candidate lists are rebuilt from these positions
  if (dyn->npm == 0) return;
  const V4<T>* __restrict__ pos = S.pos[c];
  const V4<T>* __restrict__ vel = S.vel[c];
  const V4<T>* __restrict__ idm = S.idm[c];
  const V4<T>* __restrict__ sa = S.str_a[c];
  const V2<T>* __restrict__ sb = S.str_b[c];
  const unsigned* __restrict__ nbb = S.nbb[lb];
  const V3<T> pos_i = ld3(pos, i);
  const int4 cp = S.cellpos[c][i];
  const I3 celli{cp.x, cp.y, cp.z};
  const int4 code = S.codes[c][i];
  const bool contact = code.x >= 10;
  const T th = P.two_h;
  const int cnt = live ? (dyn->list_ok ? S.nbb_cnt[lb][i] : -1) : 0;  // -1: no list, scanned
  const unsigned own = list_entry(i, kOwnCell);
  const int rounds = __reduce_max_sync(0xffffffffu, (max(cnt, 0) + kLanes - 1) / kLanes);
  // rows: s.xx s.yy s.zz kv | s.xy s.xz s.yz ker m | distance (or normal, volume) | v | rho 1
  const int y = l == 0 ? 0 : l == 1 ? 4 : l == 2 ? 8 : l == 3 ? 12 : l == 4 ? 16 : 8;
  const int x = l == 2 ? 7 : l == 5 ? 11 : 3;
  T acc[3] = {T(0), T(0), T(0)};
  int e = l, buf = 0;
  unsigned ent = group_entry(nbb, (size_t)P.npb, i, e, cnt, own);
  for (int r = 0; r < rounds; ++r, e += kLanes, buf ^= 1) {
    const int j = (int)(ent & kEntIdx);
    const int m = max(j, P.npb);  // boundary rows are written by this launch (see k_adami)
    const V4<T> pj = pos[j], vj = vel[m];
    const T mj = idm[m].y;
    const S6<T> sj = ld6(sa, sb, m);
    const V3<T> off = mulI(entry_off(ent), th);
    const bool valid = e < cnt, wall = j < P.npb;
    ent = group_entry(nbb, (size_t)P.npb, i, e + kLanes, cnt, own);
    V3<T> dr = pos_i - V3<T>{pj.x, pj.y, pj.z};
    dr = dr - off;
    const T r2 = pair_r2(dr.x, dr.y, dr.z);
    const T q = pair_r(r2) * P.i_h;
    const bool in = valid && r2 < P.r2_prefilter && q < T(2.0f);
    const T ker = kernel_w(P.knorm, q);
    const T kv = rmul(ker, mj / vj.w);
    const V3<T> gk = dr * kernel_f(P.kgrad, q);
    V4<T>* rows = sm.row[buf][warp][g];
    V4<T>* mine = rows + l * (kRow / 4);
    mine[0] = V4<T>{sj.xx, sj.yy, sj.zz, kv};
    mine[1] = V4<T>{sj.xy, sj.xz, sj.yz, ker * mj};
    mine[2] = wall ? V4<T>{gk.x, gk.y, gk.z, -P.vol_def} : V4<T>{dr.x, dr.y, dr.z, T(0)};
    mine[3] = V4<T>{vj.x, vj.y, vj.z, T(0)};
    mine[4] = V4<T>{vj.w, T(1), T(0), T(0)};
    const unsigned mat = __ballot_sync(0xffffffffu, in && !wall), nrm = __ballot_sync(0xffffffffu, in && wall);
    __syncwarp();
    group_add(rows, x, y, (l == 5 ? nrm : mat) >> (g * kLanes) & 0xffu, acc);
  }
  const int b = g * kLanes;
  const T a0 = acc[0], a1 = acc[1], a2 = acc[2];
  S6<T> rs{from_lane(a0, b), from_lane(a1, b), from_lane(a2, b), from_lane(a0, b + 1), from_lane(a1, b + 1),
           from_lane(a2, b + 1)};
  V4<T> rps{from_lane(a0, b + 2), from_lane(a1, b + 2), from_lane(a2, b + 2), from_lane(a1, b + 4)};
  V4<T> rvr{from_lane(a0, b + 3), from_lane(a1, b + 3), from_lane(a2, b + 3), from_lane(a0, b + 4)};
  V3<T> n_i{from_lane(a0, b + 5), from_lane(a1, b + 5), from_lane(a2, b + 5)};
  if (l != 0 || !live) return;
  AdamiSums<T> sums{rs, rps, rvr, n_i};
  if (cnt < 0) adami_scan<T>(P, S, c, celli, pos_i, contact, sums, nullptr);
  if (P.periodbound) {
    I3 cpb;
    V3<T> ppb;
    if (period_image(P, celli, pos_i, true, cpb, ppb)) adami_scan<T>(P, S, c, cpb, ppb, contact, sums, nullptr);
  }
  adami_finish(P, S, dyn, c, i, contact, code, pos_i, celli, sums.n_i, sums.rs, sums.rps, sums.rvr);
}

// ---------------------------------------------------------------------------------
// Nearest contact-wall particle / corner rule (src/adami_boundary.cu:209-292), plus
// the material neighbour records for the interaction.
// ---------------------------------------------------------------------------------
// Cells within one cell of a contact-wall particle (codes.x >= 10): the only cells whose
// soil particles can find a contact wall in cuFindCornerParticleMaterial's 27-cell scan.
// near_wall is cleared before each search's marking.
template <class T> __global__ void k_mark_near_wall(const Params<T> P, DevState<T> S, const Dyn<T>* dyn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.npb || !dyn->cells_dirty) return;
  const int c = dyn->cur_main;
  if (S.codes[c][i].x < 10) return;
  const int4 cp = S.cellpos[c][i];
  for (int oc = 0; oc < 27; ++oc) {
    const I3 off = off_of(oc);
    const I3 cj{cp.x + off.x, cp.y + off.y, cp.z + off.z};
    if (in_grid(P, cj)) S.near_wall[key_of(P, cj)] = 1;
  }
}

// Cells next to a marked cell (its 27-cell neighbourhood), tagged with the current
// mark generation: a list update rebuilds the lists of the particles in them.
// Grid-stride over (marked cell, neighbour) pairs.
template <class T> __global__ void k_mark_dilate(const Params<T> P, DevState<T> S, const Dyn<T>* dyn) {
  const int n = dyn->n_marks;
  if (n > RW_MARK_CAP) return;  // a full build follows
  const unsigned gen = dyn->mark_gen;
  const int ny = P.cell_num[1], nz = P.cell_num[2];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < 27 * n; k += gridDim.x * blockDim.x) {
    const int key = S.marks[k / 27];
    const I3 off = off_of(k % 27);
    const I3 cj{key / (ny * nz) + off.x, (key / nz) % ny + off.y, key % nz + off.z};
    if (in_grid(P, cj)) S.near_mark[key_of(P, cj)] = gen;
  }
}

// a.x b.x + a.y b.y + a.z b.z with fused multiply-adds at fixed places.
template <class T> RWD T dot_fma(const V3<T> a, const V3<T> b) {
  return f_fma(a.z, b.z, f_fma(a.y, b.y, rmul(a.x, b.x)));
}

// Capacity of the corner search's list of wall candidates (entries per thread).
constexpr int CORNER_THREADS = 128, CORNER_CAP = 32;
template <class T>
__global__ void __launch_bounds__(CORNER_THREADS) k_corner(const Params<T> P, DevState<T> S, const Dyn<T>* dyn,
                                                           int cpar) {
  __shared__ unsigned found_sm[CORNER_CAP][CORNER_THREADS];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int npm = dyn->npm;
  if (t >= npm) return;
  const int i = P.npb + t;
  const int c = dyn->cur_main;
  const V4<T>* __restrict__ pos = S.pos[c];
  const int4 cp = S.cellpos[c][i];
  const I3 celli{cp.x, cp.y, cp.z};
  V4<T> cv = S.cv[cpar][i];
  const bool near = P.npb > 0 && in_grid(P, celli) && S.near_wall[key_of(P, celli)];
  if (!near) {  // no contact-wall particle within the 27 cells: the scan would find nothing
    if (cv.x != T(0.0f) || cv.y != T(999)) {
      cv.x = T(0.0f);
      cv.y = T(999);
      S.cv[cpar][i] = cv;
    }
    if (dyn->rec_stale)
      write_rec(P, S.rec, i, S.pos[c][i], S.vel[c][i], ld6(S.str_a[c], S.str_b[c], i), S.idm[c][i].y,
                S.codes[c][i].x >= 10);
    return;
  }
  const V3<T> pos_i = ld3(pos, i);
  cv.x = T(0.0f);
  cv.y = T(999);
  T d_ij = T(999);
  V4<T> ny = S.cny[i];
  int nearest = -1;
  const T th = P.two_h;
  // One contact-wall candidate j at distance r = |dr|, q < 2, with normal n4 (the body of
  // the reference's scan); the nearest one's wall and velocity are read at the end.
  auto visit = [&](int j, const V3<T> dr, T r, T q, const V4<T>& n4) {
    T dwdr = kernel_f(P.kgrad, q);
    V3<T> gker = dr * dwdr;
    if (r < d_ij && r > T(0)) {
      const V3<T> n_ad{n4.x, n4.y, n4.z};
      const V3<T> n_mat = dr / r;
      d_ij = r;
      cv.y = f_abs(f_fma(dr.z, n_ad.z, f_fma(dr.x, n_ad.x, rmul(dr.y, n_ad.y))));
      nearest = j;
      const T cos_c = T(0.866f);
      const T cos_n = f_abs(dot_fma(n_mat, n_ad));
      if (cos_n < cos_c) ny = V4<T>{n_mat.x, n_mat.y, n_mat.z, T(0)};
      else ny = V4<T>{n_ad.x, n_ad.y, n_ad.z, T(0)};
    }
    cv.x += f_abs(rmul(dot_fma(xyz(ny), gker), P.vol_def));
  };
  auto offset_from = [&](const V4<T>& pj, const I3 off) {
    return pos_i - V3<T>{pj.x, pj.y, pj.z} - mulI(off, th);
  };
  // The candidate lists, current once the search has built, updated or kept them
  // (list_ok), hold every boundary particle within 2h of i in the scan's order (per cell
  // offset, the boundary range first, ascending index): walking their boundary entries
  // visits the same candidates that pass the q < 2 test, in the same order, without the
  // boundary cells' full ranges.  The boundary neighbour records (written by the Adami
  // kernel earlier in the section) carry j's position and contact flag.
  //
  // In two passes, because a warp's lanes meet their wall particles at different places of
  // their lists: taking each entry as it comes, the whole warp runs the chain of the nearest
  // particle (normal read, square root, divisions) for nearly every entry of 63 (38 us a
  // launch on the 56k-particle wall against 23, 49 against 32 at 335k, 46 against 41 at 1.92M,
  // where reading every particle's cell takes the rest).  The
  // first pass only collects the contact-wall entries within reach, eight entries' records
  // at a time; the second takes the lanes' collected entries side by side, at most some 30,
  // the next one's position and normal loaded meanwhile.  A full collection is taken and
  // emptied before the first pass goes on.
  const int kept = (S.nbg[0] && P.keep_lists && dyn->list_ok) ? S.nbg_cnt[dyn->lbuf][t] : -1;
  if (kept > 0) {
    const Rec<T>* __restrict__ rec = S.rec;
    const unsigned* __restrict__ lists = S.nbg[dyn->lbuf];
    const size_t stride = (size_t)S.nbg_stride;
    unsigned* found = &found_sm[0][threadIdx.x];
    int n = 0;
    auto take = [&] {
      V4<T> pj{T(0), T(0), T(0), T(0)}, n4 = pj;
      auto fetch = [&](int k) {
        const unsigned j = found[k * CORNER_THREADS] & kEntIdx;
        pj = rec[j].p;
        n4 = S.cny[j];
      };
      if (n > 0) fetch(0);
      for (int k = 0; k < n; ++k) {
        const unsigned ent = found[k * CORNER_THREADS];
        const V3<T> dr = offset_from(pj, entry_off(ent));
        const V4<T> nk = n4;
        if (k + 1 < n) fetch(k + 1);
        const T r = pair_r(pair_r2(dr.x, dr.y, dr.z)), q = r * P.i_h;
        if ((double)q < 2.0) visit((int)(ent & kEntIdx), dr, r, q, nk);
      }
      n = 0;
    };
    const int last_q = (kept - 1) >> 2;
    uint4 u = load_quad(lists, 0, stride, t), v = load_quad(lists, min(1, last_q), stride, t);
    for (int q0 = 0; q0 <= last_q; q0 += 2) {
      const unsigned ent[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
      V4<T> pj[8];
      T vol[8];
      bool bnd[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        bnd[k] = 4 * q0 + k < kept && (int)(ent[k] & kEntIdx) < P.npb;
        if (bnd[k]) {
          pj[k] = rec[ent[k] & kEntIdx].p;
          vol[k] = rec[ent[k] & kEntIdx].a.y;
        }
      }
      u = load_quad(lists, min(q0 + 2, last_q), stride, t);
      v = load_quad(lists, min(q0 + 3, last_q), stride, t);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const V3<T> dr = offset_from(pj[k], entry_off(ent[k]));
        if (bnd[k] && pair_r2(dr.x, dr.y, dr.z) < P.r2_prefilter && vol[k] < T(0)) {
          found[n * CORNER_THREADS] = ent[k];
          ++n;
        }
      }
      if (n > CORNER_CAP - 8) take();
    }
    take();
  } else if (kept < 0) {
    for (int oc = 0; oc < 27; ++oc) {
      const I3 off = off_of(oc);
      const I3 cj{celli.x + off.x, celli.y + off.y, celli.z + off.z};
      if (!in_grid(P, cj)) continue;
      const int2 rg = S.range[key_of(P, cj)];
      for (int j = rg.x; j < rg.y; ++j) {
        const V3<T> dr = offset_from(pos[j], off);
        const T r2 = pair_r2(dr.x, dr.y, dr.z);
        if (!(r2 < P.r2_prefilter)) continue;
        const T r = pair_r(r2), q = r * P.i_h;
        if ((double)q < 2.0 && S.codes[c][j].x >= 10) visit(j, dr, r, q, S.cny[j]);
      }
    }
  }
  V4<T> vz = S.cvz[i];
  if (nearest >= 0) {
    cv.w = (T)S.codes[c][nearest].x;
    const V4<T> vj = S.vel[c][nearest];
    vz = V4<T>{vj.x, vj.y, vj.z, T(0)};
  }
  S.cv[cpar][i] = cv;
  S.cny[i] = ny;
  S.cvz[i] = vz;
  if (dyn->rec_stale)
    write_rec(P, S.rec, i, S.pos[c][i], S.vel[c][i], ld6(S.str_a[c], S.str_b[c], i), S.idm[c][i].y,
              S.codes[c][i].x >= 10);
}

// ---------------------------------------------------------------------------------
// Particle interaction (src/particle_interaction.cu:26-297).
//
// One thread per material particle.  Phase 1 scans the 27 neighbour cells in the
// reference's order (cz, cy, cx; boundary range then material range; ascending j)
// and appends every candidate passing a conservative distance test to a per-thread
// list in shared memory (column per thread: conflict-free).  Phase 2 walks the list
// in order and evaluates the exact q < 2 test and the pair terms, so every sum is
// accumulated in the reference's order while the expensive pair arithmetic runs with
// the warp converged.  A list that fills up is flushed and the rest of the scan is
// evaluated directly, still in order.
// ---------------------------------------------------------------------------------
template <class T> struct Acc {
  T accden;
  V3<T> s, av, as;
  F9<T> gv;
};

template <class T> struct IState {
  V3<T> pos, vel;
  T rho, ri;
  S6<T> sor;
  int shift;
};


// One pair (i, j) of cuParticleInteractionMaterialLoopSolution
// (src/particle_interaction.cu:29-114), given dr = (pos_i - pos_j) - offset * 2h.
// Strict: the reference's expressions, every operation separately rounded (the CPU
// restatement's order).  Default: the same terms in fewer instructions -- r from the
// hardware reciprocal square root, the velocity-gradient products with the neighbour
// volume folded into the kernel gradient, one approximate division in the artificial
// viscosity -- a few units in the last place from the reference's roundings.
template <bool Strict, class T> RWD void pair_eval(const Params<T>& P, const IState<T>& I, const V3<T> dr,
                                                   const NbVals<T>& nb, Acc<T>& A) {
  using F = Fp<Strict>;
  const T r2 = pair_r2(dr.x, dr.y, dr.z);
  T r;
  if constexpr (Strict) r = pair_r(r2);
  else r = r2 > T(0) ? r2 * f_rsqrt(r2) : T(0);
  T q = F::mul(r, P.i_h);
  if (!(q < T(2.0f))) return;
  const T t = T(2.0f) - q;
  T dwdr = F::mul(F::mul(F::mul(P.kgrad, t), t), t);
  const V3<T> gker{F::mul(dr.x, dwdr), F::mul(dr.y, dwdr), F::mul(dr.z, dwdr)};
  const T rho_j = nb.vr.w, mass_j = nb.a.x, vol_j = f_abs(nb.a.y);
  const bool contact_j = nb.a.y < T(0);
  V3<T> dvel{I.vel.x - nb.vr.x, I.vel.y - nb.vr.y, I.vel.z - nb.vr.z};
  if (contact_j && I.shift == 1) dvel = V3<T>{T(0), T(0), T(0)};
  // grad_vel -= (dvel (x) gker) * vol_j;  accden += rho_i (dvel . gker) vol_j
  if constexpr (Strict) {
    A.gv.xx = F::msub(F::mul(dvel.x, gker.x), vol_j, A.gv.xx);
    A.gv.xy = F::msub(F::mul(dvel.x, gker.y), vol_j, A.gv.xy);
    A.gv.xz = F::msub(F::mul(dvel.x, gker.z), vol_j, A.gv.xz);
    A.gv.yx = F::msub(F::mul(dvel.y, gker.x), vol_j, A.gv.yx);
    A.gv.yy = F::msub(F::mul(dvel.y, gker.y), vol_j, A.gv.yy);
    A.gv.yz = F::msub(F::mul(dvel.y, gker.z), vol_j, A.gv.yz);
    A.gv.zx = F::msub(F::mul(dvel.z, gker.x), vol_j, A.gv.zx);
    A.gv.zy = F::msub(F::mul(dvel.z, gker.y), vol_j, A.gv.zy);
    A.gv.zz = F::msub(F::mul(dvel.z, gker.z), vol_j, A.gv.zz);
    if (contact_j) return;
    const T dvg = F::dot3(dvel.x, dvel.y, dvel.z, gker.x, gker.y, gker.z);
    A.accden = F::mad(F::mul(I.rho, dvg), vol_j, A.accden);
  } else {
    const V3<T> gkv{F::mul(gker.x, vol_j), F::mul(gker.y, vol_j), F::mul(gker.z, vol_j)};
    A.gv.xx = f_fma(-dvel.x, gkv.x, A.gv.xx);
    A.gv.xy = f_fma(-dvel.x, gkv.y, A.gv.xy);
    A.gv.xz = f_fma(-dvel.x, gkv.z, A.gv.xz);
    A.gv.yx = f_fma(-dvel.y, gkv.x, A.gv.yx);
    A.gv.yy = f_fma(-dvel.y, gkv.y, A.gv.yy);
    A.gv.yz = f_fma(-dvel.y, gkv.z, A.gv.yz);
    A.gv.zx = f_fma(-dvel.z, gkv.x, A.gv.zx);
    A.gv.zy = f_fma(-dvel.z, gkv.y, A.gv.zy);
    A.gv.zz = f_fma(-dvel.z, gkv.z, A.gv.zz);
    if (contact_j) return;
    A.accden = f_fma(I.rho, F::dot3(dvel.x, dvel.y, dvel.z, gkv.x, gkv.y, gkv.z), A.accden);
  }
  const S6<T> st{I.sor.xx + nb.a.z, I.sor.yy + nb.a.w, I.sor.zz + nb.b.x,
                 I.sor.xy + nb.b.y, I.sor.xz + nb.b.z, I.sor.yz + nb.b.w};
  const T fx = F::dot3(st.xx, st.xy, st.xz, gker.x, gker.y, gker.z);
  const T fy = F::dot3(st.xy, st.yy, st.yz, gker.x, gker.y, gker.z);
  const T fz = F::dot3(st.xz, st.yz, st.zz, gker.x, gker.y, gker.z);
  A.s.x = F::mad(fx, mass_j, A.s.x);
  A.s.y = F::mad(fy, mass_j, A.s.y);
  A.s.z = F::mad(fz, mass_j, A.s.z);
  if (P.viscosity_type == 1) {
    T artv = T(0.0f);
    const T visc = F::dot3(dvel.x, dvel.y, dvel.z, dr.x, dr.y, dr.z);
    if (visc < T(0.0f)) {
      if constexpr (Strict) {
        const T phi = F::mul(P.h, visc) / F::mad(r, r, P.eta);
        artv = F::mul(F::mul(P.alpha_m, P.cs_m), phi) / F::mul(T(0.5f), I.rho + rho_j);
      } else {  // the same quotient with one approximate division
        artv = f_fastdiv(F::mul(P.visc_k, visc), F::mul(r2 + P.eta, F::mul(T(0.5f), I.rho + rho_j)));
      }
    }
    const T m = F::mul(mass_j, artv);
    A.av.x = F::mad(gker.x, m, A.av.x);
    A.av.y = F::mad(gker.y, m, A.av.y);
    A.av.z = F::mad(gker.z, m, A.av.z);
  }
  if (P.art_coef != T(0.f)) {
    T rj = nb.a.z + nb.a.w + nb.b.x;  // artificial-stress term of j (src/particle_interaction.cu:102-104)
    if (rj > T(0.0f)) rj = F::mul(rj, P.art_coef);
    else rj = T(0.0f);
    T artp = I.ri + rj;
    if (artp > T(0.0f)) {  // W itself is only needed here (a double expression, as GetKernel)
      const T ker = kernel_w(P.knorm, q);
      artp = F::mul(artp, f_pow(ker / P.kernel_dr, P.kernel_zero / P.kernel_dr));
      const T m = F::mul(mass_j, artp);
      A.as.x = F::msub(gker.x, m, A.as.x);
      A.as.y = F::msub(gker.y, m, A.as.y);
      A.as.z = F::msub(gker.z, m, A.as.z);
    }
  }
}

// The terms of pair_eval<false>, formed without a branch, whether or not the pair counts:
// several pairs' chains (square root, division) then run side by side.
template <class T> struct PairTerms {
  V3<T> w, k, f, g;  // velocity difference, kernel gradient times volume, stress force, kernel gradient
  T q, dvk, mass, visc, mv, tr;
  bool wall;
  RWD PairTerms(const Params<T>& P, const IState<T>& I, const V3<T> dr, const NbVals<T>& nb) {
    using F = Fp<false>;
    const T r2 = pair_r2(dr.x, dr.y, dr.z);
    q = F::mul(r2 > T(0) ? r2 * f_rsqrt(r2) : T(0), P.i_h);
    const T t = T(2.0f) - q;
    const T dwdr = F::mul(F::mul(F::mul(P.kgrad, t), t), t);
    g = V3<T>{F::mul(dr.x, dwdr), F::mul(dr.y, dwdr), F::mul(dr.z, dwdr)};
    mass = nb.a.x;
    wall = nb.a.y < T(0);
    const T vol = f_abs(nb.a.y);
    w = V3<T>{I.vel.x - nb.vr.x, I.vel.y - nb.vr.y, I.vel.z - nb.vr.z};
    if (wall && I.shift == 1) w = V3<T>{T(0), T(0), T(0)};
    k = V3<T>{F::mul(g.x, vol), F::mul(g.y, vol), F::mul(g.z, vol)};
    dvk = F::dot3(w.x, w.y, w.z, k.x, k.y, k.z);
    const S6<T> st{I.sor.xx + nb.a.z, I.sor.yy + nb.a.w, I.sor.zz + nb.b.x,
                   I.sor.xy + nb.b.y, I.sor.xz + nb.b.z, I.sor.yz + nb.b.w};
    f = V3<T>{F::dot3(st.xx, st.xy, st.xz, g.x, g.y, g.z), F::dot3(st.xy, st.yy, st.yz, g.x, g.y, g.z),
              F::dot3(st.xz, st.yz, st.zz, g.x, g.y, g.z)};
    visc = F::dot3(w.x, w.y, w.z, dr.x, dr.y, dr.z);
    mv = F::mul(mass, f_fastdiv(F::mul(P.visc_k, visc), F::mul(r2 + P.eta, F::mul(T(0.5f), I.rho + nb.vr.w))));
    tr = nb.a.z + nb.a.w + nb.b.x;
  }
  // mass times the artificial stress, 0 without one
  RWD T artificial(const Params<T>& P, const IState<T>& I) const {
    using F = Fp<false>;
    if (P.art_coef == T(0.f)) return T(0);
    const T rj = tr > T(0.0f) ? F::mul(tr, P.art_coef) : T(0.0f);
    const T artp = I.ri + rj;
    if (!(artp > T(0.0f))) return T(0);
    return F::mul(mass, F::mul(artp, f_pow(kernel_w(P.knorm, q) / P.kernel_dr, P.kernel_zero / P.kernel_dr)));
  }
};

template <bool Strict, class T> RWD void pair_term(const Params<T>& P, const IState<T>& I, const V3<T> dr,
                                                   const Rec<T>* __restrict__ rec, int j, Acc<T>& A) {
  pair_eval<Strict>(P, I, dr, load_nb(rec, j), A);
}

// Particle i's own state at the start of cuParticleInteractionMaterial
// (src/particle_interaction.cu:264-277).
template <bool Strict, class T> RWD void ix_begin(const Params<T>& P, const DevState<T>& S, int c, int i,
                                                  const V4<T>& cv_i, IState<T>& I, Acc<T>& A) {
  using F = Fp<Strict>;
  I.pos = ld3(S.pos[c], i);
  const V4<T> vr_i = S.vel[c][i];
  I.vel = xyz(vr_i);
  I.rho = vr_i.w;
  I.sor = ld6(S.str_a[c], S.str_b[c], i) / F::mul(vr_i.w, vr_i.w);
  I.ri = T(0.0f);
  if (P.art_coef != T(0.f)) {
    I.ri = trace(I.sor);
    if (I.ri > T(0.0f)) I.ri = F::mul(I.ri, P.art_coef);
    else I.ri = T(0.0f);
  }
  I.shift = (int)cv_i.z;
  A.accden = T(0.f);
  A.s = A.av = A.as = V3<T>{T(0), T(0), T(0)};
  A.gv = F9<T>{T(0), T(0), T(0), T(0), T(0), T(0), T(0), T(0), T(0)};
}


// Exact float of a small integer (|v| < 2^22) without a conversion instruction.
template <class T> RWD T small_float(int v) {
  if constexpr (sizeof(T) == 4) return __int_as_float(0x4B400000 + v) - 12582912.0f;
  else return (T)v;
}

// Evaluates listed candidates of particle i in list order: a kept list (quads of list
// entries, `my` the list's first quad, `stride` columns) or the scan's shared-memory list
// (entry k at my[k * stride]: index j | offset number << 27).  The cell offset is decoded
// arithmetically (no table lookup, which would compete with the record gathers for the L1
// data stage).
template <bool Strict, class T, bool Kept = false>
RWD void ix_list_eval(const Params<T>& P, const DevState<T>& S, int c, const IState<T>& I, const unsigned* my,
                      int stride, int cnt, Acc<T>& A) {
  const Rec<T>* __restrict__ rec = S.rec;
  if (cnt <= 0) return;
  // Kept lists (global memory) are read once per interaction: streaming loads, so they
  // do not push the neighbour records out of L2.
  auto entry = [&](int k) -> unsigned {
    if constexpr (Kept) return __ldcs(my + quad_at(k >> 2, (size_t)stride, 0) + (k & 3));
    else return my[k * stride];
  };
  auto index = [](unsigned e) { return (int)(e & (Kept ? kEntIdx : 0x7ffffffu)); };
  // Entries are read two ahead and records one ahead, so a record's index is in hand
  // when its load is issued.
  unsigned ent = entry(0);
  unsigned ent1 = cnt > 1 ? entry(1) : 0u;
  unsigned oc = ent;
  NbVals<T> nb = load_nb(rec, index(ent));
#pragma unroll 2  // alternating record registers instead of copying the prefetched one
  for (int e = 0; e < cnt; ++e) {
    const NbVals<T> cur = nb;
    const unsigned occ = oc;
    if (e + 1 < cnt) {
      oc = ent1;
      nb = load_nb(rec, index(ent1));
      if (e + 2 < cnt) ent1 = entry(e + 2);
    }
    int dx, dy, dz;  // digits of the cell offset plus one (each 0..2)
    if constexpr (Kept) {
      dx = (int)(occ >> 26 & 3u);
      dy = (int)(occ >> 28 & 3u);
      dz = (int)(occ >> 30);
    } else {
      const int o = (int)(occ >> 27);
      dz = (o * 57) >> 9;
      const int rr = o - 9 * dz;
      dy = (rr * 11) >> 5;
      dx = rr - 3 * dy;
    }
    const T th = P.two_h;
    // (pos_i - p_j) - (d - 1) 2h with one rounding after the exact product: the same
    // value as subtracting the tabulated offset
    pair_eval<Strict>(P, I, V3<T>{f_fma(small_float<T>(1 - dx), th, I.pos.x - cur.p.x),
                                  f_fma(small_float<T>(1 - dy), th, I.pos.y - cur.p.y),
                                  f_fma(small_float<T>(1 - dz), th, I.pos.z - cur.p.z)}, cur, A);
  }
}

// Two floats in one 64-bit register: the packed FP32 instructions of sm_100 (each half
// rounded to nearest on its own, so a packed operation gives the two scalar results).
struct F2 {
  unsigned long long v;
};
RWD F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
RWD F2 f2(float x) { return f2(x, x); }
RWD float f2_lo(F2 a) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
  return lo;
}
RWD float f2_hi(F2 a) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
  return hi;
}
RWD F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
RWD F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
RWD F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
RWD F2 dot2(F2 ax, F2 ay, F2 az, F2 bx, F2 by, F2 bz) { return fma2(az, bz, fma2(ay, by, mul2(ax, bx))); }

RWD float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
RWD float div_ftz(float a, float b) {
  float y;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}
// f_fastdiv(a, b) for a quotient that is nearly always negative and normal: the flushing form
// then gives the same value; anything else is divided again.
RWD float div_negative(float a, float b) {
  const float y = div_ftz(a, b);
  return y <= -FLT_MIN && y >= -FLT_MAX ? y : f_fastdiv(a, b);
}

// gv -= a (x) b where ok holds.
RWD void add_grad(Acc<float>& A, float ax, float ay, float az, float bx, float by, float bz, bool ok) {
  asm("{\n\t.reg .pred p;\n\t"
      "setp.ne.s32 p, %15, 0;\n\t"
      "@p fma.rn.f32 %0, %9, %12, %0;\n\t"
      "@p fma.rn.f32 %1, %9, %13, %1;\n\t"
      "@p fma.rn.f32 %2, %9, %14, %2;\n\t"
      "@p fma.rn.f32 %3, %10, %12, %3;\n\t"
      "@p fma.rn.f32 %4, %10, %13, %4;\n\t"
      "@p fma.rn.f32 %5, %10, %14, %5;\n\t"
      "@p fma.rn.f32 %6, %11, %12, %6;\n\t"
      "@p fma.rn.f32 %7, %11, %13, %7;\n\t"
      "@p fma.rn.f32 %8, %11, %14, %8;\n\t}"
      : "+f"(A.gv.xx), "+f"(A.gv.xy), "+f"(A.gv.xz), "+f"(A.gv.yx), "+f"(A.gv.yy), "+f"(A.gv.yz), "+f"(A.gv.zx),
        "+f"(A.gv.zy), "+f"(A.gv.zz)
      : "f"(-ax), "f"(-ay), "f"(-az), "f"(bx), "f"(by), "f"(bz), "r"((int)ok));
}
// accden += rho dvk, s += f m where ok holds; av += g w where visc holds.
RWD void add_force(Acc<float>& A, float rho, float dvk, float fx, float fy, float fz, float m, float gx, float gy,
                   float gz, float w, bool ok, bool visc) {
  asm("{\n\t.reg .pred p, q;\n\t"
      "setp.ne.s32 p, %17, 0;\n\t"
      "setp.ne.s32 q, %18, 0;\n\t"
      "@p fma.rn.f32 %0, %7, %8, %0;\n\t"
      "@p fma.rn.f32 %1, %9, %12, %1;\n\t"
      "@p fma.rn.f32 %2, %10, %12, %2;\n\t"
      "@p fma.rn.f32 %3, %11, %12, %3;\n\t"
      "@q fma.rn.f32 %4, %13, %16, %4;\n\t"
      "@q fma.rn.f32 %5, %14, %16, %5;\n\t"
      "@q fma.rn.f32 %6, %15, %16, %6;\n\t}"
      : "+f"(A.accden), "+f"(A.s.x), "+f"(A.s.y), "+f"(A.s.z), "+f"(A.av.x), "+f"(A.av.y), "+f"(A.av.z)
      : "f"(rho), "f"(dvk), "f"(fx), "f"(fy), "f"(fz), "f"(m), "f"(gx), "f"(gy), "f"(gz), "f"(w), "r"((int)ok),
        "r"((int)visc));
}

// A neighbour record as its two 32-byte halves, in the order this lane reads them.
struct RawRec {
  float a[8], b[8];
};
RWD void load_half(const float* q, float (&v)[8]) {
  asm
  ("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
      : "l"(q));
}

// ix_list_eval<false, float, true> for the walk kernel, two entries at a time.  The terms
// of the two pairs are formed by packed instructions (the same operations in the same
// order as pair_eval<false>, each half rounded on its own); the sums take the entries one
// after the other, so every sum is the one ix_list_eval forms, bit for bit.  Squares that
// are then added stay scalar: the compiler fuses a packed multiply into a packed add.
//
// What bounds it: issue (61% of the cycles) and the L1 data stage (78% of its wavefronts)
// together.  The stage serves two lanes' 32-byte sectors per cycle when they lie in
// different halves of a line's 64-byte half, one otherwise (measured on random records:
// 51 cycles per warp and record pair of loads, 33 when odd lanes read the halves in the
// other order).  So odd lanes read the second half first, and the selects that put the
// halves back in order are the moves that pair the two records' fields.  Packing halves
// the issue slots of the pair terms; the packed instructions run at the FMA pipe's scalar
// rate.  1.92M-particle wall, per launch: 1.004 ms scalar, 0.955 ms packed with branches
// around the sums, 0.909 ms with predicated sums and the flushing reciprocals, 0.882 ms with
// the lists in quads (two entries a load, digits of the offset by a mask).  Scalar terms on
// the same lists: 0.903 ms (122 registers), 0.937 ms at five blocks.  The viscous quotient is
// divided with flushing first and again without where that is not normal, so that subnormal
// ones are pair_eval's: 0.855 ms with and without; unflushed for every pair 0.878, one shared
// branch for both pairs 0.960.
RWD void ix_walk_pairs(const Params<float>& P, const DevState<float>& S, const IState<float>& I,
                       const unsigned* __restrict__ lists, int t_col, size_t stride, int cnt, Acc<float>& A) {
  if (cnt <= 0) return;
  const bool odd = threadIdx.x & 1;
  const float* __restrict__ rec_a = reinterpret_cast<const float*>(S.rec) + (odd ? 8 : 0);
  const float* __restrict__ rec_b = reinterpret_cast<const float*>(S.rec) + (odd ? 0 : 8);
  const int last = (cnt - 1) & ~1;  // first entry of the last pair
  auto entries = [&](int e) {
    e = min(e, last);
    return __ldcs(reinterpret_cast<const uint2*>(lists + quad_at(e >> 2, stride, t_col) + (e & 2)));
  };
  auto load = [&](unsigned ent) {
    RawRec r;
    const size_t j = (size_t)(ent & kEntIdx) * 16;
    load_half(rec_a + j, r.a);
    load_half(rec_b + j, r.b);
    return r;
  };
  const F2 px = f2(I.pos.x), py = f2(I.pos.y), pz = f2(I.pos.z);
  const F2 vx = f2(I.vel.x), vy = f2(I.vel.y), vz = f2(I.vel.z), rho_i = f2(I.rho);
  const F2 sxx = f2(I.sor.xx), syy = f2(I.sor.yy), szz = f2(I.sor.zz), sxy = f2(I.sor.xy), sxz = f2(I.sor.xz),
           syz = f2(I.sor.yz);
  const F2 neg = f2(-1.0f), th = f2(P.two_h);
  const bool visc_on = P.viscosity_type == 1, art_on = P.art_coef != 0.0f, still = I.shift == 1;
  const bool ri_pos = I.ri > 0.0f;
  // Entries two pairs ahead, records one pair ahead.
  uint2 cur = entries(0), nxt = entries(2);
  RawRec r0 = load(cur.x), r1 = load(cur.y);
#pragma unroll 1
  for (int e = 0; e < cnt; e += 2) {
    auto lo = [&](int k) { return f2(odd ? r0.b[k] : r0.a[k], odd ? r1.b[k] : r1.a[k]); };
    auto hi = [&](int k) { return f2(odd ? r0.a[k] : r0.b[k], odd ? r1.a[k] : r1.b[k]); };
    const F2 qx = lo(0), qy = lo(1), qz = lo(2), ux = lo(4), uy = lo(5), uz = lo(6), rho_j = lo(7);
    const F2 mass = hi(0), svol = hi(1), jxx = hi(2), jyy = hi(3), jzz = hi(4), jxy = hi(5), jxz = hi(6), jyz = hi(7);
    const unsigned c0 = cur.x >> 26, c1 = cur.y >> 26;
    cur = nxt;
    r0 = load(cur.x);
    r1 = load(cur.y);
    nxt = entries(e + 4);
    // dr = (pos_i - p_j) - offset 2h.  A digit d masked in place (d << s) and or-ed into
    // the bits of 3 2^22 is the float 3 2^22 + (d << s); one exact multiply-add makes it
    // 1 - d, and the product with 2h is exact: one rounding.
    auto digit = [&](unsigned mask, float scale) {
      const F2 f = f2(__uint_as_float((c0 & mask) | 0x4B400000u), __uint_as_float((c1 & mask) | 0x4B400000u));
      return fma2(f, f2(-scale), f2(12582912.0f * scale + 1.0f));
    };
    const F2 dx = fma2(digit(3u, 1.0f), th, fma2(qx, neg, px));
    const F2 dy = fma2(digit(12u, 0.25f), th, fma2(qy, neg, py));
    const F2 dz = fma2(digit(48u, 0.0625f), th, fma2(qz, neg, pz));
    const float ra = pair_r2(f2_lo(dx), f2_lo(dy), f2_lo(dz)), rb = pair_r2(f2_hi(dx), f2_hi(dy), f2_hi(dz));
    const F2 r2 = f2(ra, rb);
    // r = r2 / sqrt(r2); below the floor, 2 - q is 2 as at r2 = 0
    const float ma = f_max(ra, 1e-30f), mb = f_max(rb, 1e-30f);
    const F2 r = f2(ma * rsqrt_ftz(ma), mb * rsqrt_ftz(mb));
    const F2 q = mul2(r, f2(P.i_h));
    const bool ok0 = f2_lo(q) < 2.0f, ok1 = f2_hi(q) < 2.0f && e + 1 < cnt;
    const F2 t = fma2(q, neg, f2(2.0f));
    const F2 dwdr = mul2(mul2(mul2(f2(P.kgrad), t), t), t);
    const F2 gx = mul2(dx, dwdr), gy = mul2(dy, dwdr), gz = mul2(dz, dwdr);
    const float v0 = f2_lo(svol), v1 = f2_hi(svol);
    const bool con0 = v0 < 0.0f, con1 = v1 < 0.0f;
    F2 wx = fma2(ux, neg, vx), wy = fma2(uy, neg, vy), wz = fma2(uz, neg, vz);
    if (still) {  // no velocity difference against a contact wall
      wx = f2(con0 ? 0.0f : f2_lo(wx), con1 ? 0.0f : f2_hi(wx));
      wy = f2(con0 ? 0.0f : f2_lo(wy), con1 ? 0.0f : f2_hi(wy));
      wz = f2(con0 ? 0.0f : f2_lo(wz), con1 ? 0.0f : f2_hi(wz));
    }
    const F2 vol = f2(f_abs(v0), f_abs(v1));
    const F2 kx = mul2(gx, vol), ky = mul2(gy, vol), kz = mul2(gz, vol);
    const F2 dvk = dot2(wx, wy, wz, kx, ky, kz);
    const F2 txx = add2(sxx, jxx), tyy = add2(syy, jyy), tzz = add2(szz, jzz);
    const F2 txy = add2(sxy, jxy), txz = add2(sxz, jxz), tyz = add2(syz, jyz);
    const F2 fx = dot2(txx, txy, txz, gx, gy, gz);
    const F2 fy = dot2(txy, tyy, tyz, gx, gy, gz);
    const F2 fz = dot2(txz, tyz, tzz, gx, gy, gz);
    const F2 vd = dot2(wx, wy, wz, dx, dy, dz);
    const F2 num = mul2(f2(P.visc_k), vd);
    const F2 den = mul2(add2(r2, f2(P.eta)), mul2(f2(0.5f), add2(rho_i, rho_j)));
    const F2 artv = f2(f2_lo(vd) < 0.0f ? div_negative(f2_lo(num), f2_lo(den)) : 0.0f,
                       f2_hi(vd) < 0.0f ? div_negative(f2_hi(num), f2_hi(den)) : 0.0f);
    const F2 mv = mul2(mass, artv);
    const F2 tr = add2(add2(jxx, jyy), jzz);
    // the sums of one pair, predicated instead of branched over (a lane or two of a warp
    // usually has a candidate between 2h and the list radius)
    auto sums = [&](auto half, bool ok, bool con) {
      add_grad(A, half(wx), half(wy), half(wz), half(kx), half(ky), half(kz), ok);
      add_force(A, I.rho, half(dvk), half(fx), half(fy), half(fz), half(mass), half(gx), half(gy), half(gz),
                half(mv), ok && !con, ok && !con && visc_on);
      if (art_on && ok && !con && (ri_pos || half(tr) > 0.0f)) {  // artificial stress, as in pair_eval
        float rj = half(tr);
        rj = rj > 0.0f ? __fmul_rn(rj, P.art_coef) : 0.0f;
        float artp = I.ri + rj;
        if (artp > 0.0f) {
          const float ker = kernel_w(P.knorm, half(q));
          artp = __fmul_rn(artp, f_pow(ker / P.kernel_dr, P.kernel_zero / P.kernel_dr));
          const float w = __fmul_rn(half(mass), artp);
          A.as.x = f_fma(-half(gx), w, A.as.x);
          A.as.y = f_fma(-half(gy), w, A.as.y);
          A.as.z = f_fma(-half(gz), w, A.as.z);
        }
      }
    };
    sums([](F2 v) { return f2_lo(v); }, ok0, con0);
    sums([](F2 v) { return f2_hi(v); }, ok1, con1);
  }
}

// Pair sums of particle i straight from global memory: phase 1 lists candidates in
// shared memory (my[k * stride]), phase 2 evaluates them in order.  A list that fills
// up is evaluated and emptied, and the scan resumes (order preserved).
template <bool Strict, class T> RWD void ix_sums_global(const Params<T>& P, const DevState<T>& S, int c, const I3 celli,
                                                        const IState<T>& I, unsigned* my, int stride, int cap,
                                                        Acc<T>& A) {
  const V4<T>* __restrict__ pos = S.pos[c];
  const T th = P.two_h;
  const T r2max = P.r2_prefilter;
  int cnt = 0;
  for (int oc = 0; oc < 27; ++oc) {
    const I3 off = off_of(oc);
    const I3 cj{celli.x + off.x, celli.y + off.y, celli.z + off.z};
    if (!in_grid(P, cj)) continue;
    const int k = key_of(P, cj);
    const V3<T> pmo = I.pos - mulI(off, th);  // conservative pre-test only
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      const int2 rg = S.range[pass ? k + P.ncell_material : k];
#pragma unroll 4
      for (int j = rg.x; j < rg.y; ++j) {
        const V4<T> pj = pos[j];
        const T dx = pmo.x - pj.x, dy = pmo.y - pj.y, dz = pmo.z - pj.z;
        if (dx * dx + dy * dy + dz * dz < r2max) {
          if (cnt == cap) {
            ix_list_eval<Strict>(P, S, c, I, my, stride, cnt, A);
            cnt = 0;
          }
          my[cnt * stride] = (unsigned)j | ((unsigned)oc << 27);
          ++cnt;
        }
      }
    }
  }
  ix_list_eval<Strict>(P, S, c, I, my, stride, cnt, A);
}

// Second pass of a particle within 2h of a periodic plane, over the neighbours of its
// periodic image (cuParticleInteractionMaterialLoopPeriod,
// src/particle_interaction.cu:243-257): same order, evaluated directly (few particles).
template <bool Strict, class T> RWD void ix_period(const Params<T>& P, const DevState<T>& S, int c, int i,
                                                   const I3 celli, IState<T>& I, Acc<T>& A) {
  I3 cpb;
  V3<T> ppb;
  if (!period_image(P, celli, I.pos, false, cpb, ppb)) return;
  const V4<T>* __restrict__ pos = S.pos[c];
  const V3<T> keep = I.pos;
  I.pos = ppb;
  for (int oc = 0; oc < 27; ++oc) {
    const I3 off = off_of(oc);
    const I3 cj{cpb.x + off.x, cpb.y + off.y, cpb.z + off.z};
    if (!in_grid(P, cj)) continue;
    const int k = key_of(P, cj);
    const V3<T> o = mulI(off, P.two_h);
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      const int2 rg = S.range[pass ? k + P.ncell_material : k];
#pragma unroll 1
      for (int j = rg.x; j < rg.y; ++j) {
        const V4<T> pj = pos[j];
        pair_term<Strict>(P, I, I.pos - V3<T>{pj.x, pj.y, pj.z} - o, S.rec, j, A);
      }
    }
  }
  I.pos = keep;
}

// End of cuParticleInteractionMaterial: provisional velocity, wall contact
// (cuParticleInteractionMaterialLoopContact, src/particle_interaction.cu:142-241) and
// the stage outputs (src/particle_interaction.cu:284-295).
template <bool Strict, class T> RWD void ix_finish(const Params<T>& P, const DevState<T>& S, int c, int cpar, int i,
                                                   const I3 celli, const IState<T>& I, const Acc<T>& A, V4<T> cv) {
  using F = Fp<Strict>;
  const V4<T>* __restrict__ cv_in = S.cv[cpar];
  const V4<T>* __restrict__ cf_in = S.cf[cpar];
  const V3<T> g{P.gravity[0], P.gravity[1], P.gravity[2]};
  const V3<T> damp{F::mul(I.vel.x, P.damping), F::mul(I.vel.y, P.damping), F::mul(I.vel.z, P.damping)};
  const V3<T> acc0{A.s.x + A.av.x + A.as.x - damp.x + g.x, A.s.y + A.av.y + A.as.y - damp.y + g.y,
                   A.s.z + A.av.z + A.as.z - damp.z + g.z};
  const V4<T> vr_new{F::mad(acc0.x, P.dt, I.vel.x), F::mad(acc0.y, P.dt, I.vel.y), F::mad(acc0.z, P.dt, I.vel.z),
                     F::mad(A.accden, P.dt, I.rho)};
  V3<T> acc_st{T(0.0f), T(0.0f), T(0.0f)};
  V4<T> fo = cf_in[i];
  const V4<T> ny = S.cny[i];
  const V4<T> vz = S.cvz[i];
  const T mass_i = S.idm[c][i].y;
  const T mrate = T(2.0f) / (T(2.0f) + T(0.0f));
  const V3<T> dv{F::mul(vz.x - vr_new.x, mrate), F::mul(vz.y - vr_new.y, mrate), F::mul(vz.z - vr_new.z, mrate)};
  const T dvn_s = F::dot3(dv.x, dv.y, dv.z, ny.x, ny.y, ny.z);
  if (cv.y <= F::mul(P.h, T(2)) && dvn_s > T(0)) {
    const T fcoef = P.wall_fric;
    const V3<T> dvn{F::mul(ny.x, dvn_s), F::mul(ny.y, dvn_s), F::mul(ny.z, dvn_s)};
    const V3<T> fn{F::mul(dvn.x, mass_i) / P.dt, F::mul(dvn.y, mass_i) / P.dt, F::mul(dvn.z, mass_i) / P.dt};
    const V3<T> dvt{dv.x - dvn.x, dv.y - dvn.y, dv.z - dvn.z};
    V3<T> ft{F::mul(dvt.x, mass_i) / P.dt, F::mul(dvt.y, mass_i) / P.dt, F::mul(dvt.z, mass_i) / P.dt};
    const T afn = f_sqrt(F::dot3(fn.x, fn.y, fn.z, fn.x, fn.y, fn.z));
    const T aft = f_sqrt(F::dot3(ft.x, ft.y, ft.z, ft.x, ft.y, ft.z));
    const T cap = F::mul(fcoef, afn);
    if (aft > cap) {
      const T ratio = cap / aft;
      ft = V3<T>{F::mul(ft.x, ratio), F::mul(ft.y, ratio), F::mul(ft.z, ratio)};
      cv.z = T(1);
    } else {
      cv.z = T(0);
    }
    V3<T> fric{ft.x + fn.x, ft.y + fn.y, ft.z + fn.z};
    if (cv.y > F::mul(P.dr, T(1.0f))) {
      // The reference walks the soil of the 27 cells in order, takes the smallest kernel
      // integral met so far and lets each particle met replace the friction: what remains is
      // the smallest of all and the friction of the last one in that order (offset number,
      // then index).  So the order of the visits is free: the three cells of a z column are
      // one run of indices, its distances are read sixteen at a time and the particles next
      // to the wall among them four at a time.  One load per particle, each waited for, took
      // most of a small case's launch (56k-particle wall: the walk 96 us, 50 now; 1.92M: 0.875 ms, 0.859).
      const T h2 = F::mul(T(2.0f), P.h);
      const V3<T> pabs_i{F::mad((T)celli.x, h2, I.pos.x), F::mad((T)celli.y, h2, I.pos.y),
                         F::mad((T)celli.z, h2, I.pos.z)};
      const T ylim = F::mul(P.dr, T(1.0001f));
      const T half_dr = P.dr / T(2);
      long long last = -1;  // offset number << 32 | index of the last one met
      T last_x = T(0);
      auto meet = [&](int j, const V4<T>& pj, const int4& cpj, T cvx, int col) {
        const V3<T> pabs_j{F::mad((T)cpj.x, h2, pj.x), F::mad((T)cpj.y, h2, pj.y), F::mad((T)cpj.z, h2, pj.z)};
        const V3<T> dc{pabs_i.x - pabs_j.x, pabs_i.y - pabs_j.y, pabs_i.z - pabs_j.z};
        const T rcol = f_abs(F::dot3(dc.x, dc.y, dc.z, ny.z, ny.y, ny.x));
        const T x = j == i ? cv.x : cvx;
        if (!(rcol <= half_dr && x != T(0))) return;
        if (cv.x > x) cv.x = x;
        const long long key = ((long long)(col + 9 * (cpj.z - celli.z + 1)) << 32) | j;
        if (key > last) {
          last = key;
          last_x = cvx;
        }
      };
      for (int col = 0; col < 9; ++col) {
        const int cx = celli.x + col % 3 - 1, cy = celli.y + col / 3 - 1;
        if (cx < 0 || cy < 0 || cx >= P.cell_num[0] || cy >= P.cell_num[1]) continue;
        const int k0 = P.ncell_material + key_of(P, I3{cx, cy, 0});
        int beg = INT_MAX, end = 0;
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz) {
          const int cz = celli.z + dz;
          const int2 rg = cz >= 0 && cz < P.cell_num[2] ? S.range[k0 + cz] : int2{0, 0};
          if (rg.y > rg.x) {
            beg = min(beg, rg.x);
            end = max(end, rg.y);
          }
        }
        for (int j0 = beg; j0 < end; j0 += 16) {
          unsigned near = 0;
#pragma unroll
          for (int k = 0; k < 16; ++k) near |= (cv_in[min(j0 + k, end - 1)].y <= ylim ? 1u : 0u) << k;
          if (end - j0 < 16) near &= (1u << (end - j0)) - 1u;
          while (near) {
            int jj[4];
            V4<T> pj[4];
            int4 cpj[4];
            T xj[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              jj[k] = near ? j0 + __ffs(near) - 1 : -1;
              near &= near - 1u;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int j = jj[k] >= 0 ? jj[k] : jj[0];
              pj[k] = S.pos[c][j];
              cpj[k] = S.cellpos[c][j];
              xj[k] = cv_in[j].x;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (jj[k] >= 0) meet(jj[k], pj[k], cpj[k], xj[k], col);
          }
        }
      }
      if (last >= 0) {
        const int j = (int)(last & 0x7fffffff);
        const T x = j == i ? cv.x : last_x;
        const V4<T> fj = cf_in[j];
        fric = V3<T>{F::mul(fj.x, cv.x) / x, F::mul(fj.y, cv.x) / x, F::mul(fj.z, cv.x) / x};
      } else {
        fric = V3<T>{F::mul(fric.x, T(0)), F::mul(fric.y, T(0)), F::mul(fric.z, T(0))};
      }
    }
    fo = V4<T>{fric.x, fric.y, fric.z, T(0)};
    const T im = T(1) / mass_i;
    acc_st = V3<T>{F::mul(fric.x, im), F::mul(fric.y, im), F::mul(fric.z, im)};
  }
  S.cv[cpar ^ 1][i] = cv;
  S.cf[cpar ^ 1][i] = fo;
  S.accad[i] = V4<T>{A.s.x + A.av.x + A.as.x + acc_st.x - damp.x + g.x, A.s.y + A.av.y + A.as.y + acc_st.y - damp.y + g.y,
                     A.s.z + A.av.z + A.as.z + acc_st.z - damp.z + g.z, A.accden};
  st6(S.ace_a, S.ace_b, i, full2sym(A.gv));
  S.spin[i] = v4(skewpart(A.gv), T(0.f));
}

// Candidate lists of the live soil particles: the 27 cells in the scan's order (cz,
// cy, cx; boundary range before material range; ascending j), every candidate within
// the list radius, written column-major to HBM.  Mode 0 builds every soil list here and
// starts the displacement bounds (the Adami kernel builds the boundary lists).  Mode 2
// (list update) queues the lists of particles next to a marked cell, soil and boundary
// rows alike, for k_rebuild_lists, and carries the others through the section's
// permutation; the bounds run on from the last full build (a list built since then
// moved no more than its particle's bound).  A list longer than IX_CAP is marked -1 and
// counted (n_spill): the scan launch then takes that particle.  Light (no pair
// arithmetic, no shared-memory list), so it runs at full occupancy; the walk kernel
// then evaluates the lists with the same pairs in the same order as a scan.  One thread
// per particle, boundary rows first, so that in an update the Adami kernel (many
// registers, few warps per SM) only walks lists.
template <class T>
__global__ void __launch_bounds__(256) k_build_lists(const Params<T> P, DevState<T> S, Dyn<T>* dyn, int bnd) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  const int mode = dyn->ix_mode;
  if (!S.nbg[0] || !P.keep_lists || mode == 1) return;
  if (row == 0 && mode == 0) {
    dyn->list_ok = 1;
    dyn->list_kill = dyn->build_kill;
  }
  const int lb = dyn->lbuf;
  const int c = dyn->cur_main;
  // queues a row whose list k_rebuild_lists rebuilds (one warp per list), so that the
  // few lists an update rebuilds do not each wait on one thread's 27-cell scan
  auto enqueue = [&] {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&dyn->n_queue, __popc(m));
    base = __shfl_sync(m, base, leader);
    S.queue[base + __popc(m & ((1u << lane) - 1u))] = row;
  };
  if (row < P.npb) {
    if (mode == 0 && bnd) enqueue();
    if (mode == 2 && S.nbb[0]) {
      const int4 cb = S.cellpos[c][row];
      if (near_marked(P, S, dyn, I3{cb.x, cb.y, cb.z})) enqueue();
      else if (dyn->need_sort)
        carry_list(S.nbb[lb ^ 1], S.nbb_cnt[lb ^ 1], S.sperm[row], S.nbb[lb], S.nbb_cnt[lb], row, P.npb, S.inv);
    }
    return;
  }
  const int t = row - P.npb;
  if (t >= dyn->npm) return;
  const int i = row;
  const int4 cp = S.cellpos[c][i];
  const I3 celli{cp.x, cp.y, cp.z};
  const size_t stride = (size_t)S.nbg_stride;
  if (mode == 2) {
    if (!near_marked(P, S, dyn, celli)) {
      if (dyn->need_sort)
        carry_list(S.nbg[lb ^ 1], S.nbg_cnt[lb ^ 1], S.sperm[i] - P.npb, S.nbg[lb], S.nbg_cnt[lb], t, stride, S.inv);
      return;
    }
    enqueue();  // next to a marked cell
    return;
  }
  S.dacc[lb][i] = 0.0f;
  const V4<T>* __restrict__ pos = S.pos[c];
  const V3<T> pos_i = ld3(pos, i);
  const T th = P.two_h;
  QuadWriter out{S.nbg[lb], stride, t};
  for (int oc = 0; oc < 27; ++oc) {
    const I3 off = off_of(oc);
    const I3 cj{celli.x + off.x, celli.y + off.y, celli.z + off.z};
    if (!in_grid(P, cj)) continue;
    const int k = key_of(P, cj);
    const unsigned code = list_entry(0, oc);
    const V3<T> pmo = pos_i - mulI(off, th);  // conservative pre-test only
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      const int2 rg = S.range[pass ? k + P.ncell_material : k];
#pragma unroll 4
      for (int j = rg.x; j < rg.y; ++j) {
        const V4<T> pj = pos[j];
        const T dx = pmo.x - pj.x, dy = pmo.y - pj.y, dz = pmo.z - pj.z;
        if (dx * dx + dy * dy + dz * dz < P.r2_list) out.push((unsigned)j | code, IX_CAP);
      }
    }
  }
  out.finish(list_entry(i, kOwnCell), IX_CAP);
  const int cnt = out.cnt;
  if (cnt > IX_CAP) {
    S.nbg_cnt[lb][t] = -1;
    atomicAdd(&dyn->n_spill, 1);
  } else {
    S.nbg_cnt[lb][t] = cnt;
  }
}

// The lists queued by a list update (soil rows' interaction lists and boundary rows'
// Adami lists; in a full build with eight lanes per particle, every boundary row's), one
// warp per list: the 27 cells x 2 ranges are 54 segments of
// candidates, flattened in the scan's order; the warp tests 32 consecutive candidates
// at a time and appends the hits in order (ballot + prefix count), so the list holds
// the pairs a full build lists, in the same order.  The displacement bounds run on.
template <class T> __global__ void __launch_bounds__(256) k_rebuild_lists(const Params<T> P, DevState<T> S, Dyn<T>* dyn) {
  constexpr int kSeg = 54, kWarps = 256 / 32;
  __shared__ int seg_beg[kWarps][kSeg + 1];  // first flattened candidate of each segment
  __shared__ int seg_j0[kWarps][kSeg];       // first particle index of each segment
  if (!S.nbg[0] || !P.keep_lists || dyn->ix_mode == 1) return;
  const int nq = dyn->n_queue;
  if (blockIdx.x == 0 && threadIdx.x == 0 && dyn->ix_mode == 2) dyn->n_rebuilt += nq;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lb = dyn->lbuf, c = dyn->cur_main;
  const V4<T>* __restrict__ pos = S.pos[c];
  const T th = P.two_h;
  int* beg = seg_beg[warp];
  int* j0 = seg_j0[warp];
  for (int q = blockIdx.x * kWarps + warp; q < nq; q += gridDim.x * kWarps) {
    // a soil row's list, or a boundary row's Adami list (without the boundary ranges
    // unless the particle belongs to a contact wall, as the Adami scan keeps it)
    const int i = S.queue[q];
    const bool bnd = i < P.npb;
    const bool with_bnd_range = !bnd || S.codes[c][i].x >= 10;
    const int4 cp = S.cellpos[c][i];
    const I3 celli{cp.x, cp.y, cp.z};
    const V3<T> pos_i = ld3(pos, i);
    int size[2], first[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int sg = lane + 32 * h;
      size[h] = 0;
      first[h] = 0;
      if (sg < kSeg && ((sg & 1) || with_bnd_range)) {
        const I3 off = off_of(sg >> 1);
        const I3 cj{celli.x + off.x, celli.y + off.y, celli.z + off.z};
        if (in_grid(P, cj)) {
          const int k = key_of(P, cj);
          const int2 rg = S.range[(sg & 1) ? k + P.ncell_material : k];
          size[h] = rg.y - rg.x;
          first[h] = rg.x;
        }
      }
    }
    int inc0 = size[0], inc1 = size[1];  // inclusive prefix sums over the lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, inc0, d), b = __shfl_up_sync(0xffffffffu, inc1, d);
      if (lane >= d) {
        inc0 += a;
        inc1 += b;
      }
    }
    const int tot0 = __shfl_sync(0xffffffffu, inc0, 31);
    const int total = tot0 + __shfl_sync(0xffffffffu, inc1, 31);
    beg[lane] = inc0 - size[0];
    j0[lane] = first[0];
    if (lane + 32 < kSeg) {
      beg[lane + 32] = tot0 + inc1 - size[1];
      j0[lane + 32] = first[1];
    }
    if (lane == 0) beg[kSeg] = total;
    __syncwarp();
    const size_t stride = bnd ? (size_t)P.npb : (size_t)S.nbg_stride;
    unsigned* __restrict__ out = bnd ? S.nbb[lb] : S.nbg[lb];
    const int col = bnd ? i : i - P.npb;
    int* __restrict__ count = bnd ? S.nbb_cnt[lb] + i : S.nbg_cnt[lb] + (i - P.npb);
    int cnt = 0;
    for (int b0 = 0; b0 < total; b0 += 32) {
      const int ci = b0 + lane;
      bool hit = false;
      unsigned ent = 0u;
      if (ci < total) {
        int lo = 0, hi = kSeg;  // the last segment starting at or before ci (it is not empty)
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (beg[mid] <= ci) lo = mid;
          else hi = mid;
        }
        const int j = j0[lo] + (ci - beg[lo]);
        const int oc = lo >> 1;
        const V3<T> pmo = pos_i - mulI(off_of(oc), th);
        const V4<T> pj = pos[j];
        const T dx = pmo.x - pj.x, dy = pmo.y - pj.y, dz = pmo.z - pj.z;
        hit = dx * dx + dy * dy + dz * dz < P.r2_list;
        ent = list_entry(j, oc);
      }
      const unsigned bal = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int e = cnt + __popc(bal & ((1u << lane) - 1u));
        if (e < IX_CAP) __stcs(out + quad_at(e >> 2, stride, col) + (e & 3), ent);
      }
      cnt += __popc(bal);
    }
    if (cnt < IX_CAP && lane < (-cnt & 3))  // fill up the last quad
      __stcs(out + quad_at(cnt >> 2, stride, col) + (cnt & 3) + lane, list_entry(i, kOwnCell));
    if (lane == 0) {
      *count = cnt > IX_CAP ? -1 : cnt;  // an overflowed boundary list: Adami scans for it
      if (cnt > IX_CAP && !bnd) atomicAdd(&dyn->n_spill, 1);
    }
    __syncwarp();  // before the next list overwrites the segment table
  }
}

// Interaction, one thread per soil particle, neighbours read from global memory, as
// two launches that split the particles between them:
//  - walk (Walk = true): walks the candidate lists, kept from an earlier section or
//    just built by k_build_lists.  It carries no scan state, so it runs with fewer
//    registers;
//  - scan (Walk = false): scans the 27 cells for the particles without a list (lists
//    off, or a list that overflowed) and carries the contact state of deleted slots.
// The packed walk holds two records ahead and two in use: 128 registers, four blocks of
// 128 threads per SM (five blocks spill: 1.83 ms per launch against 0.91).
template <class T, bool Strict> constexpr bool kPackedWalk = !Strict && sizeof(T) == 4;
template <class T, bool Strict, bool Walk>
__global__ void __launch_bounds__(Walk ? IX_WALK_MAX_THREADS : IX_THREADS, Walk && kPackedWalk<T, Strict> ? 4 : 0)
    k_interaction(const Params<T> P, DevState<T> S, const Dyn<T>* dyn, int cpar) {
  extern __shared__ unsigned nbl[];  // IX_CAP x blockDim, column per thread (scan only)
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (!Walk && t == 0) const_cast<Dyn<T>*>(dyn)->rec_stale = 0;  // the corner search has refreshed the records
  const int total = P.np - P.npb;
  if (t >= total) return;
  const int i = P.npb + t;
  const int npm = dyn->npm;
  const bool keep = S.nbg[0] && P.keep_lists;
  if (Walk) {
    if (!keep || t >= npm) return;
  } else if (t >= npm) {  // deleted slots keep their contact state
    S.cv[cpar ^ 1][i] = S.cv[cpar][i];
    S.cf[cpar ^ 1][i] = S.cf[cpar][i];
    return;
  }
  const int lb = dyn->lbuf;
  const int kept = keep ? S.nbg_cnt[lb][t] : -1;
  if (Walk != (kept >= 0)) return;  // the other launch takes this particle
  const int c = dyn->cur_main;
  const int4 cp = S.cellpos[c][i];
  const I3 celli{cp.x, cp.y, cp.z};
  const V4<T> cv = S.cv[cpar][i];
  IState<T> I;
  Acc<T> A;
  ix_begin<Strict>(P, S, c, i, cv, I, A);
  if constexpr (Walk && kPackedWalk<T, Strict>) ix_walk_pairs(P, S, I, S.nbg[lb], t, (size_t)S.nbg_stride, kept, A);
  else if (Walk) ix_list_eval<Strict, T, true>(P, S, c, I, S.nbg[lb] + (size_t)4 * t, S.nbg_stride, kept, A);
  else ix_sums_global<Strict>(P, S, c, celli, I, nbl + threadIdx.x, blockDim.x, IX_CAP, A);
  if (P.periodbound) ix_period<Strict>(P, S, c, i, celli, I, A);
  ix_finish<Strict>(P, S, c, cpar, i, celli, I, A, cv);
}

// The walk with eight lanes per particle (see GroupRows), for cases that a thread per particle
// leaves waiting.  The terms are pair_eval<false>'s; lanes 0..2 add the rows of the velocity
// gradient, 3 the stress force, 4 the viscous one, 5 the artificial stress, 6 the density rate.
// 693-particle column 15 us a launch against 28, 5.4k in FP64 32 against 54.  What bounds it
// when it fills the GPU is the L1 data stage (73% of its wavefronts at 28k): per eight
// entries the rows cost as many again as the record gathers, so beyond some 16k particles
// the thread per particle is faster (41 us against 36 at 28k).
template <class T>
__global__ void __launch_bounds__(kGroupThreads) k_interaction_group(const Params<T> P, DevState<T> S, const Dyn<T>* dyn,
                                                                     int cpar) {
  __shared__ GroupRows<T> sm;
  const int lane = threadIdx.x & 31, l = lane & (kLanes - 1), g = lane / kLanes, warp = threadIdx.x >> 5;
  const int t0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  const int npm = dyn->npm, lb = dyn->lbuf, c = dyn->cur_main;
  if (npm == 0) return;
  const int t = min(t0, npm - 1), i = P.npb + t;
  const int kept = t0 < npm ? S.nbg_cnt[lb][t] : -1;  // -1: the scan launch takes this particle
  const int cnt = max(kept, 0);
  const int rounds = __reduce_max_sync(0xffffffffu, (cnt + kLanes - 1) / kLanes);
  const V4<T> cv = S.cv[cpar][i];
  IState<T> I;
  Acc<T> A;
  ix_begin<false>(P, S, c, i, cv, I, A);
  const Rec<T>* __restrict__ rec = S.rec;
  const unsigned* __restrict__ lists = S.nbg[lb];
  const size_t stride = (size_t)S.nbg_stride;
  const unsigned own = list_entry(i, kOwnCell);
  const T th = P.two_h;
  // rows: k.x k.y k.z -w.x | f.x f.y f.z -w.y | g.x g.y g.z -w.z | dvk 0 0 mass | mv -ma rho_i 0
  const int y = l < 3 ? 0 : l == 3 ? 4 : l < 6 ? 8 : 12;
  const int x = l < 3 ? 3 + 4 * l : l == 3 ? 15 : l < 6 ? 12 + l : 18;
  T acc[3] = {T(0), T(0), T(0)};
  int e = l, buf = 0;
  unsigned ent = group_entry(lists, stride, t, e, cnt, own), nxt = group_entry(lists, stride, t, e + kLanes, cnt, own);
  NbVals<T> nb = load_nb(rec, (int)(ent & kEntIdx));
  for (int r = 0; r < rounds; ++r, e += kLanes, buf ^= 1) {
    const NbVals<T> cur = nb;
    const I3 off = entry_off(ent);
    ent = nxt;
    nb = load_nb(rec, (int)(ent & kEntIdx));
    nxt = group_entry(lists, stride, t, e + 2 * kLanes, cnt, own);
    const V3<T> dr{f_fma((T)-off.x, th, I.pos.x - cur.p.x), f_fma((T)-off.y, th, I.pos.y - cur.p.y),
                   f_fma((T)-off.z, th, I.pos.z - cur.p.z)};
    const PairTerms<T> p(P, I, dr, cur);
    const bool in = e < cnt && p.q < T(2.0f), wall = p.wall;
    const T ma = in && !wall ? p.artificial(P, I) : T(0);
    V4<T>* rows = sm.row[buf][warp][g];
    V4<T>* mine = rows + l * (kRow / 4);
    mine[0] = V4<T>{p.k.x, p.k.y, p.k.z, -p.w.x};
    mine[1] = V4<T>{p.f.x, p.f.y, p.f.z, -p.w.y};
    mine[2] = V4<T>{p.g.x, p.g.y, p.g.z, -p.w.z};
    mine[3] = V4<T>{p.dvk, T(0), T(0), p.mass};
    mine[4] = V4<T>{p.mv, -ma, I.rho, T(0)};
    const unsigned b_in = __ballot_sync(0xffffffffu, in), b_mat = __ballot_sync(0xffffffffu, in && !wall);
    const unsigned b_visc = __ballot_sync(0xffffffffu, in && !wall && p.visc < T(0.0f) && P.viscosity_type == 1);
    const unsigned b_art = __ballot_sync(0xffffffffu, ma != T(0));
    const unsigned on = l < 3 ? b_in : l == 4 ? b_visc : l == 5 ? b_art : b_mat;
    __syncwarp();
    group_add(rows, x, y, on >> (g * kLanes) & 0xffu, acc);
  }
  const int b = g * kLanes;
  const T a0 = acc[0], a1 = acc[1], a2 = acc[2];
  A.gv = F9<T>{from_lane(a0, b), from_lane(a1, b), from_lane(a2, b), from_lane(a0, b + 1), from_lane(a1, b + 1),
               from_lane(a2, b + 1), from_lane(a0, b + 2), from_lane(a1, b + 2), from_lane(a2, b + 2)};
  A.s = V3<T>{from_lane(a0, b + 3), from_lane(a1, b + 3), from_lane(a2, b + 3)};
  A.av = V3<T>{from_lane(a0, b + 4), from_lane(a1, b + 4), from_lane(a2, b + 4)};
  A.as = V3<T>{from_lane(a0, b + 5), from_lane(a1, b + 5), from_lane(a2, b + 5)};
  A.accden = from_lane(a0, b + 6);
  if (l != 0 || kept < 0) return;
  const int4 cp = S.cellpos[c][i];
  const I3 celli{cp.x, cp.y, cp.z};
  if (P.periodbound) ix_period<false>(P, S, c, i, celli, I, A);
  ix_finish<false>(P, S, c, cpar, i, celli, I, A, cv);
}

// ---------------------------------------------------------------------------------
// Chunked interaction with the neighbour tile staged in shared memory.
//
// The soil particles of one cell column (x, y) are contiguous and ordered by z, so a
// chunk of up to IX2_TB of them needs the 9 columns (x+-1, y+-1) over the z window
// [z_first - 1, z_last + 1], in both layers: 18 contiguous index runs.  The block
// copies those runs' positions into shared memory once; every candidate test of
// phase 1 then reads shared memory.  Lists are filled in warp-synchronous rounds of
// IX2_CAP entries (a round ends for the whole warp when any lane's list is full) and
// evaluated in order with the next neighbour record prefetched, so each particle's
// sums keep the reference's order exactly.  A chunk whose tile does not fit
// (more than IX2_SMAX particles or IX2_NZW cells in z) runs the global path.
// ---------------------------------------------------------------------------------
constexpr int IX2_TB = 128, IX2_SMAX = 2048, IX2_NZW = 30, IX2_CAP = 96;

// Run of a staged index: boundary runs are staged before material runs, so the layer
// is k >= base of the first material run; the column comes from the cell offset.
RWD int ix2_seg(int k, int oc, int base9) {
  const I3 off = off_of(oc);
  return (k >= base9 ? 9 : 0) + (off.y + 1) * 3 + (off.x + 1);
}

struct Chunk {
  int first, n, col, pad;
};

template <class T> struct Ix2Smem {
  V4<T> spos[IX2_SMAX];
  int2 tab[18][IX2_NZW];
  int delta[18];   // global index = staged index + delta
  int gbeg[18], glen[18], base[18];
  unsigned short list[IX2_CAP][IX2_TB];  // staged index (11 bits) | cell offset << 11
  int zl, nzw, total, fallback;
};

// Per-column soil runs and chunk counts (the chunk list is rebuilt after each sort).
template <class T> __global__ void k_col_count(const Params<T> P, DevState<T> S) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  const int ncol = P.cell_num[0] * P.cell_num[1];
  if (col >= ncol) return;
  const int nz = P.cell_num[2];
  const int base = P.ncell_material + col * nz;
  int beg = -1, end = -1;
  for (int z = 0; z < nz; ++z) {
    const int2 r = S.range[base + z];
    if (r.y > r.x) {
      if (beg < 0) beg = r.x;
      end = r.y;
    }
  }
  const int len = beg < 0 ? 0 : end - beg;
  S.col_beg[col] = beg < 0 ? 0 : beg;
  S.col_len[col] = len;
  S.col_cnt[col] = (len + IX2_TB - 1) / IX2_TB;
}

template <class T> __global__ void __launch_bounds__(1024) k_col_scan(const Params<T> P, DevState<T> S, Dyn<T>* dyn) {
  __shared__ int ws[32];
  const int ncol = P.cell_num[0] * P.cell_num[1];
  const int per = (ncol + 1023) / 1024;
  const int b = threadIdx.x * per, e = min(ncol, b + per);
  int s = 0;
  for (int k = b; k < e; ++k) s += S.col_cnt[k];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = s;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[w] = x;
  __syncthreads();
  if (w == 0) {
    int v = ws[lane];
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += y;
    }
    ws[lane] = v;
  }
  __syncthreads();
  int off = x - s + (w > 0 ? ws[w - 1] : 0);
  for (int k = b; k < e; ++k) {
    const int n = S.col_cnt[k];
    S.col_off[k] = off;
    off += n;
  }
  if (threadIdx.x == 1023) dyn->nchunks = off;
}

template <class T> __global__ void k_col_fill(const Params<T> P, DevState<T> S) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  const int ncol = P.cell_num[0] * P.cell_num[1];
  if (col >= ncol) return;
  const int n = S.col_cnt[col];
  if (n == 0) return;
  const int len = S.col_len[col], beg = S.col_beg[col], off = S.col_off[col];
  for (int k = 0; k < n; ++k) {  // n nearly equal chunks
    const int a = beg + (int)((long)len * k / n);
    const int b = beg + (int)((long)len * (k + 1) / n);
    S.chunks[off + k] = Chunk{a, b - a, col, 0};
  }
}

template <class T, bool Strict> __global__ void __launch_bounds__(IX2_TB) k_interaction2(const Params<T> P, DevState<T> S,
                                                                                       const Dyn<T>* dyn, int cpar) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Ix2Smem<T>& sm = *reinterpret_cast<Ix2Smem<T>*>(smraw);
  const int tid = threadIdx.x;
  if (blockIdx.x == 0 && tid == 0) const_cast<Dyn<T>*>(dyn)->rec_stale = 0;  // records refreshed by the corner search
  // Deleted slots keep their contact state (the chunk list covers live particles only).
  {
    const int npm = dyn->npm;
    const int ndel = P.np - P.npb - npm;
    for (int t = blockIdx.x * IX2_TB + tid; t < ndel; t += gridDim.x * IX2_TB) {
      const int i = P.npb + npm + t;
      S.cv[cpar ^ 1][i] = S.cv[cpar][i];
      S.cf[cpar ^ 1][i] = S.cf[cpar][i];
    }
  }
  if ((int)blockIdx.x >= dyn->nchunks) return;
  const Chunk ch = S.chunks[blockIdx.x];
  const int c = dyn->cur_main;
  const int ny = P.cell_num[1], nz = P.cell_num[2];
  const int x = ch.col / ny, y = ch.col % ny;
  if (tid == 0) {
    const int z0 = S.cellpos[c][ch.first].z;
    const int z1 = S.cellpos[c][ch.first + ch.n - 1].z;
    const int zl = max(z0 - 1, 0), zh = min(z1 + 1, nz - 1);
    sm.zl = zl;
    sm.nzw = zh - zl + 1;
  }
  __syncthreads();
  const int zl = sm.zl, nzw = sm.nzw;
  const bool fits_z = nzw <= IX2_NZW;
  if (fits_z) {
    // Cell table (global ranges for now) of the 18 runs.
    for (int idx = tid; idx < 18 * nzw; idx += IX2_TB) {
      const int s = idx / nzw, zi = idx - s * nzw;
      const int lay = s / 9, c9 = s - lay * 9;
      const int xx = x + c9 % 3 - 1, yy = y + c9 / 3 - 1;
      int2 r{0, 0};
      if (xx >= 0 && yy >= 0 && xx < P.cell_num[0] && yy < ny)
        r = S.range[(lay ? P.ncell_material : 0) + xx * ny * nz + yy * nz + zl + zi];
      sm.tab[s][zi] = r;
    }
  }
  __syncthreads();
  if (tid < 18) {
    int gb = 0, ge = 0;
    bool any = false;
    if (fits_z)
      for (int zi = 0; zi < nzw; ++zi) {
        const int2 r = sm.tab[tid][zi];
        if (r.y > r.x) {
          if (!any) gb = r.x;
          ge = r.y;
          any = true;
        }
      }
    sm.gbeg[tid] = gb;
    sm.glen[tid] = any ? ge - gb : 0;
  }
  __syncthreads();
  if (tid == 0) {
    int tot = 0;
    for (int s = 0; s < 18; ++s) {
      sm.base[s] = tot;
      sm.delta[s] = sm.gbeg[s] - tot;
      tot += sm.glen[s];
    }
    sm.total = tot;
    sm.fallback = (!fits_z || tot > IX2_SMAX) ? 1 : 0;
  }
  __syncthreads();
  const bool fallback = sm.fallback != 0;
  if (!fallback) {
    // Staged coordinates for the table; copy the runs' positions.
    for (int idx = tid; idx < 18 * nzw; idx += IX2_TB) {
      const int s = idx / nzw, zi = idx - s * nzw;
      const int2 r = sm.tab[s][zi];
      sm.tab[s][zi] = (r.y > r.x) ? int2{r.x - sm.delta[s], r.y - sm.delta[s]} : int2{0, 0};
    }
    const V4<T>* __restrict__ pos = S.pos[c];
    for (int s = 0; s < 18; ++s) {
      const int n = sm.glen[s], gb = sm.gbeg[s], b = sm.base[s];
      for (int k = tid; k < n; k += IX2_TB) sm.spos[b + k] = pos[gb + k];
    }
  }
  __syncthreads();
  if (tid >= ch.n) return;
  const int i = ch.first + tid;
  const int4 cp = S.cellpos[c][i];
  const I3 celli{cp.x, cp.y, cp.z};
  const V4<T> cv = S.cv[cpar][i];
  IState<T> I;
  Acc<T> A;
  ix_begin<Strict>(P, S, c, i, cv, I, A);
  if (fallback) {
    // Too big for the tile: same arithmetic from global memory, list in the round buffer.
    ix_sums_global<Strict>(P, S, c, celli, I, reinterpret_cast<unsigned*>(&sm.list[0][0]) + tid, IX2_TB,
                           IX2_CAP / 2, A);
    if (P.periodbound) ix_period<Strict>(P, S, c, i, celli, I, A);
    ix_finish<Strict>(P, S, c, cpar, i, celli, I, A, cv);
    return;
  }
  const Rec<T>* __restrict__ rec = S.rec;
  const T th = P.two_h;
  const T r2max = P.r2_prefilter;
  const int zi_i = cp.z - zl;
  const unsigned lanes = __activemask();
  unsigned short* my = &sm.list[0][tid];
  int cnt = 0;
  // Evaluate the listed candidates in order (next neighbour record prefetched).
  auto flush = [&]() {
    if (cnt > 0) {
      int kk = my[0] & 0x7ff, oc = my[0] >> 11;
      NbVals<T> nb = load_nb(rec, kk + sm.delta[ix2_seg(kk, oc, sm.base[9])]);
      for (int e = 0; e < cnt; ++e) {
        const NbVals<T> cur = nb;
        const int kc = kk, occ = oc;
        if (e + 1 < cnt) {
          const unsigned short ent = my[(e + 1) * IX2_TB];
          kk = ent & 0x7ff;
          oc = ent >> 11;
          nb = load_nb(rec, kk + sm.delta[ix2_seg(kk, oc, sm.base[9])]);
        }
        const V3<T> o = mulI(off_of(occ), th);
        const V4<T> pj = sm.spos[kc];
        pair_eval<Strict>(P, I, I.pos - V3<T>{pj.x, pj.y, pj.z} - o, cur, A);
      }
    }
    cnt = 0;
  };
  // Phase 1 over the 54 (cell offset, layer) ranges in the reference's order; a range
  // that could overflow any lane's list first flushes every lane's list.
  for (int oc = 0; oc < 27; ++oc) {
    const I3 off = off_of(oc);
    const int zz = zi_i + off.z;
    const bool zin = zz >= 0 && zz < nzw;
    const V3<T> pmo = I.pos - mulI(off, th);
#pragma unroll 1
    for (int lay = 0; lay < 2; ++lay) {
      int2 r{0, 0};
      if (zin) r = sm.tab[lay * 9 + (off.y + 1) * 3 + (off.x + 1)][zz];
      if (__any_sync(lanes, cnt + (r.y - r.x) > IX2_CAP)) flush();
      for (int k = r.x; k < r.y; ++k) {
        const V4<T> pj = sm.spos[k];
        const T dx = pmo.x - pj.x, dy = pmo.y - pj.y, dz = pmo.z - pj.z;
        if (dx * dx + dy * dy + dz * dz < r2max) {
          if (cnt == IX2_CAP) flush();  // only a cell with more than IX2_CAP particles gets here
          my[cnt * IX2_TB] = (unsigned short)(k | (oc << 11));
          ++cnt;
        }
      }
    }
  }
  flush();
  if (P.periodbound) ix_period<Strict>(P, S, c, i, celli, I, A);
  ix_finish<Strict>(P, S, c, cpar, i, celli, I, A, cv);
}

// ---------------------------------------------------------------------------------
// What an integrator reads of its rows: the state's own arrays (row i at [i]) or a block's
// rows staged in shared memory (row of thread t at [t]).
// ---------------------------------------------------------------------------------
template <class T> struct RowIn {
  const V4<T>*pos, *vel, *sa, *na;  // predictor: the state; corrector: the step-start state
  const V4<T>*idm, *acc, *da, *spin, *po, *kp, *kv;
  const V2<T>*sb, *nb, *db;
  const int4 *codes, *cell;
  const float* dacc;
};
template <class T, int Stage> RWD RowIn<T> row_in(const DevState<T>& S, const Dyn<T>* dyn) {
  const int c = dyn->cur_main, ci = dyn->cur_ini;
  RowIn<T> r;
  r.pos = Stage == 0 ? S.pos[c] : S.pos_ini[ci];
  r.vel = Stage == 0 ? S.vel[c] : S.vel_ini[ci];
  r.sa = Stage == 0 ? S.str_a[c] : S.stri_a[ci];
  r.sb = Stage == 0 ? S.str_b[c] : S.stri_b[ci];
  r.na = Stage == 0 ? S.stn_a[c] : S.stni_a[ci];
  r.nb = Stage == 0 ? S.stn_b[c] : S.stni_b[ci];
  r.kp = Stage == 0 ? S.cmp_p[c] : S.cmp_pi[ci];
  r.kv = Stage == 0 ? S.cmp_v[c] : S.cmp_vi[ci];
  r.idm = S.idm[c];
  r.acc = S.accad;
  r.da = S.ace_a;
  r.db = S.ace_b;
  r.spin = S.spin;
  r.codes = S.codes[c];
  r.cell = S.cellpos[c];
  r.po = S.pos_ori[c];
  r.dacc = S.dacc[dyn->lbuf];
  return r;
}
// Bytes a staged row takes.
template <class T> constexpr int staged_row_bytes(int stage, bool mixed) {
  const int v4 = 8 + (stage == 1) + (mixed ? 2 : 0);
  return v4 * (int)sizeof(V4<T>) + 3 * (int)sizeof(V2<T>) + (1 + (stage == 1)) * (int)sizeof(int4) + (int)sizeof(float);
}
// Fetches the block's rows [i0, i0 + blockDim.x) into shared memory with one bulk copy per
// array and points `in` at them; false if they did not arrive (the caller then reads the
// state's arrays, and waits once more before it ends).  Every array starts on a 256-byte
// boundary and i0 is a multiple of the block, so a copy starts and ends on 16 bytes.
template <class T, int Stage>
RWD bool stage_rows(const Params<T>& P, int i0, unsigned char* raw, uint64_t* bar, RowIn<T>& in) {
  const int nt = blockDim.x;
  if (threadIdx.x == 0) {
    tc::mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::mbar_expect(bar, (uint32_t)(nt * staged_row_bytes<T>(Stage, P.mixed != 0)));
  }
  int off = 0;
  auto put = [&](auto*& p) {
    const int bytes = nt * (int)sizeof(*p);
    if (threadIdx.x == 0) tc::bulk_load(raw + off, p + i0, (uint32_t)bytes, bar);
    p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(raw + off);
    off += bytes;
  };
  put(in.pos);
  put(in.vel);
  put(in.codes);
  put(in.sa);
  put(in.na);
  put(in.acc);
  put(in.da);
  put(in.spin);
  put(in.idm);
  if (Stage == 1) {
    put(in.cell);
    put(in.po);
  }
  if (P.mixed) {
    put(in.kp);
    put(in.kv);
  }
  put(in.sb);
  put(in.nb);
  put(in.db);
  put(in.dacc);
  __syncthreads();
  return __syncthreads_and(tc::mbar_wait(bar, 0));
}

// ---------------------------------------------------------------------------------
// Predictor (src/predictor_corrector.cu:52-103): saves the step-start state into the
// *_ini buffers (the reference's four D2D copies) and advances material half a step.
// ---------------------------------------------------------------------------------
// Both integrators stream about 400 B per particle.  Read directly, the predictor waits on
// memory in four dependent turns (its step-start stores hold the later loads back): four
// 256-thread blocks per SM, 64 registers, 172 us at 1.9M particles, 4.6 TB/s.  With its rows
// staged by bulk copies it waits once, the step-start copies leave from shared memory, and
// three blocks (80 registers, 32 spilled bytes) take 140 us, 5.7 TB/s (four blocks: 149, two
// without spills: 170); fetching the next blocks' rows into L2 ahead only adds (152).
// In FP64 four blocks spill 500 to 800 bytes; two (128 registers) take 18 us instead of 26 at
// 60k particles and 28 instead of 31 to 33 at 112k (three: 23 and 28, one: 23 and 34).
// One row of the predictor, read at in[k]; Saved: the step-start copies are made elsewhere.
// With the learned closure on, HypoCS rows keep their stress here and the closure's pass
// updates it (and writes their record).
template <bool Saved, class T>
RWD void predictor_row(const Params<T>& P, const DevState<T>& S, const Dyn<T>* dyn, int i, const RowIn<T>& in, int k) {
  if (i >= P.np) return;
  const int c = dyn->cur_main, ci = dyn->cur_ini;
  const int npm = dyn->npm;
  V4<T> ps = in.pos[k];
  V4<T> vr = in.vel[k];
  if (!Saved) {
    S.pos_ini[ci][i] = ps;
    S.vel_ini[ci][i] = vr;
  }
  V4<T> kp{T(0), T(0), T(0), T(0)}, kv{T(0), T(0), T(0), T(0)};
  if (P.mixed) {
    kp = in.kp[k];
    kv = in.kv[k];
    if (!Saved) {
      S.cmp_pi[ci][i] = kp;
      S.cmp_vi[ci][i] = kv;
    }
  }
  if (npm == 0 || i >= P.npb + npm) return;
  S6<T> sg = ld6(in.sa, in.sb, k);
  S6<T> sn = ld6(in.na, in.nb, k);
  if (!Saved) {
    st6(S.stri_a[ci], S.stri_b[ci], i, sg);
    st6(S.stni_a[ci], S.stni_b[ci], i, sn);
  }
  if (i < P.npb) return;
  const int4 code = in.codes[k];
  if (code.y != 1) return;
  const T mass = in.idm[k].y;  // for the neighbour record (read early: the stores below may alias)
  const T hdt = T(0.5f) * P.dt;
  const V4<T> acc = in.acc[k];
  if (P.mixed) {  // compensated half step; the compensation itself is not kept
    kahan_add(vr.x, kv.x, acc.x * hdt);
    kahan_add(vr.y, kv.y, acc.y * hdt);
    kahan_add(vr.z, kv.z, acc.z * hdt);
    kahan_add(vr.w, kv.w, acc.w * hdt);
    kahan_add(ps.x, kp.x, vr.x * hdt);
    kahan_add(ps.y, kp.y, vr.y * hdt);
    kahan_add(ps.z, kp.z, vr.z * hdt);
  } else {
    vr = vr + acc * hdt;
    ps = add3(ps, xyz(vr) * hdt);
  }
  {  // distance since the lists were built, after this half step
    const float a = (float)(f_sqrt(vr.x * vr.x + vr.y * vr.y + vr.z * vr.z) * hdt);
    if (in.dacc[k] + a + P.disp_eps > P.disp_lim) const_cast<Dyn<T>*>(dyn)->list_kill = 1;
  }
  const T* mp = P.model_par[code.w];
  vr.w = f_max(vr.w, mp[kMatSize - 2]);
  vr.w = f_min(vr.w, mp[kMatSize - 1]);
  const S6<T> D = ld6(in.da, in.db, k);
  sn = sn + D * hdt;
  bool yld = false;
  T mcrt = T(0);
  const bool by_closure = P.closure && code.z == RW_MODEL_HYPO_CS;  // the closure pass updates the stress
  const HypoC<T> hc = P.hypo[code.w];
  if (!by_closure) constitutive(code.z, mp, hdt, vr.w, xyz(in.spin[k]), D, sg, yld, mcrt, P.mixed != 0, &hc);
  S.pos[c][i] = ps;
  S.vel[c][i] = vr;
  st6(S.stn_a[c], S.stn_b[c], i, sn);
  st6(S.str_a[c], S.str_b[c], i, sg);
  if (!yld) S.idm[c][i].x = T(100);
  if (!by_closure) write_rec(P, S.rec, i, ps, vr, sg, mass, code.x >= 10);
}

template <class T, bool Staged>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? (Staged ? 3 : 4) : 2)
    k_predictor(const Params<T> P, DevState<T> S, const Dyn<T>* dyn) {
  const int i0 = blockIdx.x * blockDim.x, tid = threadIdx.x;
  const RowIn<T> in = row_in<T, 0>(S, dyn);
  if constexpr (Staged) {
    extern __shared__ __align__(128) unsigned char raw[];
    __shared__ uint64_t bar;
    if (i0 >= P.npb && i0 + (int)blockDim.x <= P.npb + dyn->npm) {  // block-uniform
      RowIn<T> st = in;
      if (stage_rows<T, 0>(P, i0, raw, &bar, st)) {
        if (tid == 0) {  // the step-start copies leave from the staged rows
          const int ci = dyn->cur_ini, n4 = blockDim.x * (int)sizeof(V4<T>), n2 = blockDim.x * (int)sizeof(V2<T>);
          tc::bulk_store(S.pos_ini[ci] + i0, st.pos, n4);
          tc::bulk_store(S.vel_ini[ci] + i0, st.vel, n4);
          tc::bulk_store(S.stri_a[ci] + i0, st.sa, n4);
          tc::bulk_store(S.stri_b[ci] + i0, st.sb, n2);
          tc::bulk_store(S.stni_a[ci] + i0, st.na, n4);
          tc::bulk_store(S.stni_b[ci] + i0, st.nb, n2);
          if (P.mixed) {
            tc::bulk_store(S.cmp_pi[ci] + i0, st.kp, n4);
            tc::bulk_store(S.cmp_vi[ci] + i0, st.kv, n4);
          }
          tc::bulk_store_commit();
        }
        predictor_row<true>(P, S, dyn, i0 + tid, st, tid);
        if (tid == 0) tc::bulk_store_wait();
        return;
      }
      tc::mbar_wait(&bar, 0);  // late: read the arrays instead, with no copy left in flight
    }
  }
  predictor_row<false>(P, S, dyn, i0 + tid, in, i0 + tid);
}

// ---------------------------------------------------------------------------------
// Corrector (src/predictor_corrector.cu:109-213): rigid walls and material.
// ---------------------------------------------------------------------------------
// Rounding error of s = fl(a + b): exact(a + b) - s (Knuth's TwoSum).
template <class T> RWD T two_sum_err(T a, T b, T s) {
  const T bb = add_rn(s, -a);
  return add_rn(add_rn(a, -add_rn(s, -bb)), add_rn(b, -bb));
}

template <class T> RWD I3 rebin(V4<T>& ps, T th) {
  I3 dc{int(ps.x >= th) - int(ps.x < T(0)), int(ps.y >= th) - int(ps.y < T(0)), int(ps.z >= th) - int(ps.z < T(0))};
  ps = sub3(ps, mulI(dc, th));
  return dc;
}

// Marks a cell whose particles changed (once per generation: the first marker lists it).
template <class T> RWD void mark_cell(const Params<T>& P, const DevState<T>& S, const Dyn<T>* dyn, I3 c) {
  const int key = key_of(P, c);
  const unsigned gen = dyn->mark_gen;
  if (atomicExch(&S.cell_mark[key], gen) != gen) {
    const int k = atomicAdd(&const_cast<Dyn<T>*>(dyn)->n_marks, 1);
    if (k < RW_MARK_CAP) S.marks[k] = key;
  }
}

// Bookkeeping of the kept candidate lists for one particle's full step from cell `from`
// to cell `to`.  Its distance bound grows by the step (plus a rounding allowance) and
// must stay within the skin's share, else every list is rebuilt.  A cell change marks
// both cells (the next list update rebuilds the lists around them); leaving the grid
// (deletion) makes it a full build.
template <class T> RWD void list_account(const Params<T>& P, const DevState<T>& S, const Dyn<T>* dyn, int i, float dacc,
                                         float step, I3 from, I3 to) {
  const float d = dacc + step + P.disp_eps;
  S.dacc[dyn->lbuf][i] = d;
  Dyn<T>* w = const_cast<Dyn<T>*>(dyn);
  if (from.x != to.x || from.y != to.y || from.z != to.z) {
    w->cells_dirty = 1;
    if (!in_grid(P, from) || !in_grid(P, to)) {
      w->list_kill = 1;
    } else if (P.keep_lists) {
      mark_cell(P, S, dyn, from);
      mark_cell(P, S, dyn, to);
    }
  }
  if (d > P.disp_lim) w->list_kill = 1;
}

// One row of the corrector (moving boundary rows and soil rows); with the learned
// closure on, HypoCS rows keep their stress here, as in predictor_row.
template <class T>
RWD void corrector_row(const Params<T>& P, const DevState<T>& S, const Dyn<T>* dyn, int i, const RowIn<T>& in, int k) {
  const int npm = dyn->npm;
  if (i >= P.npb + npm) return;
  const int c = dyn->cur_main;
  const int4 code = in.codes[k];
  if (code.y != 1) return;
  const T th = P.two_h;
  if (i < P.npb) {
    if (P.n_motion <= 0) return;
    const Motion<T>& mv = dyn->mv[code.w];
    V3<T> vel{mv.trans_vel.x, mv.trans_vel.y, mv.trans_vel.z};
    int4 cp = in.cell[k];
    if (mv.is_rotat && mv.pattern != RW_PATTERN_CIRCLE) {
      const V3<T> pabs = ld3(S.pos[c], i) + mulI(I3{cp.x, cp.y, cp.z}, th);
      const V3<T> rp{mv.pos_rp.x, mv.pos_rp.y, mv.pos_rp.z};
      const V3<T> w{mv.rotat_vel.x, mv.rotat_vel.y, mv.rotat_vel.z};
      vel = vel + cross(w, pabs - rp);
      const F9<T> R = rodrigues(w * P.dt);
      const int cn = dyn->cur_nrm;
      const V4<T> n4 = S.normal[cn][i];
      const V3<T> n = dotFV(R, xyz(n4));
      S.normal[cn][i] = v4(n, n4.w);
    }
    V4<T> ps = add3(in.pos[k], vel * P.dt);
    const I3 dc = rebin(ps, th);
    S.pos[c][i] = ps;
    S.cellpos[c][i] = int4{cp.x + dc.x, cp.y + dc.y, cp.z + dc.z, cp.w};
    list_account(P, S, dyn, i, in.dacc[k], (float)(f_sqrt(dot(vel, vel)) * P.dt), I3{cp.x, cp.y, cp.z},
                 I3{cp.x + dc.x, cp.y + dc.y, cp.z + dc.z});
    return;
  }
  const V4<T> vri = in.vel[k];
  V4<T> id = in.idm[k];  // read early: the stores below may alias
  V4<T> vr, ps;
  V4<T> kp{T(0), T(0), T(0), T(0)}, kv{T(0), T(0), T(0), T(0)};
  if (P.mixed) {  // compensated full step (position and velocity keep their lost low bits)
    kp = in.kp[k];
    kv = in.kv[k];
    const V4<T> acc = in.acc[k];
    vr = vri;
    kahan_add(vr.x, kv.x, acc.x * P.dt);
    kahan_add(vr.y, kv.y, acc.y * P.dt);
    kahan_add(vr.z, kv.z, acc.z * P.dt);
    kahan_add(vr.w, kv.w, acc.w * P.dt);
    ps = in.pos[k];
    const T hdt = T(0.5f) * P.dt;
    kahan_add(ps.x, kp.x, (vr.x + vri.x) * hdt);
    kahan_add(ps.y, kp.y, (vr.y + vri.y) * hdt);
    kahan_add(ps.z, kp.z, (vr.z + vri.z) * hdt);
  } else {
    vr = vri + in.acc[k] * P.dt;
    ps = add3(in.pos[k], xyz(vr + vri) * (T(0.5f) * P.dt));
  }
  const T* mp = P.model_par[code.w];
  vr.w = f_max(vr.w, mp[kMatSize - 2]);
  vr.w = f_min(vr.w, mp[kMatSize - 1]);
  const V4<T> ps0 = ps;
  const I3 dc = rebin(ps, th);
  if (P.mixed) {  // re-binning adds -+2h: fold its rounding error into the compensation
    const V3<T> sh = mulI(dc, th);
    kp.x = add_rn(kp.x, -two_sum_err(ps0.x, -sh.x, ps.x));
    kp.y = add_rn(kp.y, -two_sum_err(ps0.y, -sh.y, ps.y));
    kp.z = add_rn(kp.z, -two_sum_err(ps0.z, -sh.z, ps.z));
    S.cmp_p[c][i] = kp;
    S.cmp_v[c][i] = kv;
  }
  const int4 cp0 = in.cell[k];
  int4 cp = int4{cp0.x + dc.x, cp0.y + dc.y, cp0.z + dc.z, cp0.w};
  if (P.periodbound) period_wrap(P, cp, ps);
  {
    const V3<T> inc = xyz(vr + vri) * (T(0.5f) * P.dt);
    list_account(P, S, dyn, i, in.dacc[k], (float)f_sqrt(dot(inc, inc)), I3{cp0.x, cp0.y, cp0.z}, I3{cp.x, cp.y, cp.z});
  }
  S6<T> sg = ld6(in.sa, in.sb, k);
  const S6<T> D = ld6(in.da, in.db, k);
  const S6<T> sn = ld6(in.na, in.nb, k) + D * P.dt;
  bool yld = false;
  T mcrt = T(0);
  const bool by_closure = P.closure && code.z == RW_MODEL_HYPO_CS;  // the closure pass updates the stress
  const HypoC<T> hc = P.hypo[code.w];
  if (!by_closure) constitutive(code.z, mp, P.dt, vr.w, xyz(in.spin[k]), D, sg, yld, mcrt, P.mixed != 0, &hc);
  if (!yld) id.x = T(100);
  id.w = mcrt;
  if (!in_grid(P, I3{cp.x, cp.y, cp.z})) {
    cp.w = P.ncell_delete_m;
    id.x = T(999.0);
  }
  V4<T> po = in.po[k];
  if (dyn->time_f <= P.dt) po = V4<T>{T(0), T(0), T(0), T(0)};
  po = add3(po, xyz(vr) * P.dt);
  S.vel[c][i] = vr;
  S.pos[c][i] = ps;
  S.cellpos[c][i] = cp;
  st6(S.str_a[c], S.str_b[c], i, sg);
  st6(S.stn_a[c], S.stn_b[c], i, sn);
  S.idm[c][i] = id;
  S.pos_ori[c][i] = po;
  S.accad[i] = po;
  if (!by_closure) write_rec(P, S.rec, i, ps, vr, sg, id.y, code.x >= 10);
}

template <class T, bool Staged>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? (Staged ? 3 : 4) : 2)
    k_corrector(const Params<T> P, DevState<T> S, const Dyn<T>* dyn) {
  const int i0 = blockIdx.x * blockDim.x, tid = threadIdx.x;
  const RowIn<T> in = row_in<T, 1>(S, dyn);
  if constexpr (Staged) {
    extern __shared__ __align__(128) unsigned char raw[];
    __shared__ uint64_t bar;
    if (i0 >= P.npb && i0 + (int)blockDim.x <= P.npb + dyn->npm) {  // block-uniform
      RowIn<T> st = in;
      if (stage_rows<T, 1>(P, i0, raw, &bar, st)) {
        corrector_row(P, S, dyn, i0 + tid, st, tid);
        return;
      }
      tc::mbar_wait(&bar, 0);
    }
  }
  corrector_row(P, S, dyn, i0 + tid, in, i0 + tid);
}

// ---------------------------------------------------------------------------------
// Shepard stress filter (src/field_smoothing.cu:26-111).  store != 0 copies the
// result back into the stress (StressRegularization) and refreshes the records.
// ---------------------------------------------------------------------------------
template <class T> __global__ void __launch_bounds__(128) k_shepard(const Params<T> P, DevState<T> S, const Dyn<T>* dyn,
                                                                   int only_filter_steps) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int npm = dyn->npm;
  if (t >= npm) return;
  if (only_filter_steps) {
    const int st = dyn->step;
    if (!(P.stress_shepard_filter != 0 && st % P.stress_shepard_filter == 0 && st != 0)) return;
  }
  const int i = P.npb + t;
  const int c = dyn->cur_main;
  const V4<T>* __restrict__ pos = S.pos[c];
  const V3<T> pos_i = ld3(pos, i);
  const int4 cp = S.cellpos[c][i];
  const I3 celli{cp.x, cp.y, cp.z};
  S6<T> sh = zero6<T>();
  T sumker = T(0.0f);
  const T th = P.two_h;
  auto scan = [&](const I3 cc, const V3<T> pp) {
    for (int oc = 0; oc < 27; ++oc) {
      const I3 off = off_of(oc);
      const I3 cj{cc.x + off.x, cc.y + off.y, cc.z + off.z};
      if (!in_grid(P, cj)) continue;
      const int2 rg = S.range[key_of(P, cj) + P.ncell_material];
      const V3<T> o = mulI(off, th);
      for (int j = rg.x; j < rg.y; ++j) {
        V3<T> dr = pp - ld3(pos, j) - o;
        const T r2 = pair_r2(dr.x, dr.y, dr.z);
        if (!(r2 < P.r2_prefilter)) continue;
        T r = pair_r(r2);
        T q = r * P.i_h;
        if (q < T(2.0f)) {
          T ker = kernel_w(P.knorm, q);
          T vol = S.idm[c][j].y / S.vel[c][j].w;
          sumker += ker * vol;
          sh = sh + ld6(S.str_a[c], S.str_b[c], j) * (ker * vol);
        }
      }
    }
  };
  // Inside the step (only_filter_steps) the filter runs after the corner search, where
  // the candidate lists are current (built, updated or kept at the end of the search)
  // and so are the neighbour records.  A list holds every material neighbour within
  // 2h in the scan's order (per cell offset, ascending index): walking its material
  // entries, with position, density and volume from the records, visits the same pairs
  // in the same order.  Entries four at a time, their data loaded together.
  const int kept = (only_filter_steps && S.nbg[0] && P.keep_lists && dyn->list_ok) ? S.nbg_cnt[dyn->lbuf][t] : -1;
  if (kept >= 0) {
    const Rec<T>* __restrict__ rec = S.rec;
    const unsigned* __restrict__ lists = S.nbg[dyn->lbuf];
    const size_t stride = (size_t)S.nbg_stride;
    constexpr unsigned kNone = kEntIdx;
    for (int e0 = 0; e0 < kept; e0 += 4) {
      unsigned ent[4];
      NbVals<T> nb[4];
      S6<T> sj[4];
      const uint4 q = load_quad(lists, e0 >> 2, stride, t);
      ent[0] = q.x;
      ent[1] = e0 + 1 < kept ? q.y : kNone;
      ent[2] = e0 + 2 < kept ? q.z : kNone;
      ent[3] = e0 + 3 < kept ? q.w : kNone;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int j = (int)(ent[k] & kNone);
        if (j == (int)kNone || j < P.npb) continue;
        nb[k] = load_nb(rec, j);
        sj[k] = ld6(S.str_a[c], S.str_b[c], j);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int j = (int)(ent[k] & kNone);
        if (j == (int)kNone || j < P.npb) continue;
        V3<T> dr = pos_i - V3<T>{nb[k].p.x, nb[k].p.y, nb[k].p.z};
        dr = dr - mulI(entry_off(ent[k]), th);
        const T r2 = pair_r2(dr.x, dr.y, dr.z);
        if (!(r2 < P.r2_prefilter)) continue;
        T r = pair_r(r2);
        T q = r * P.i_h;
        if (q < T(2.0f)) {
          T ker = kernel_w(P.knorm, q);
          T vol = f_abs(nb[k].a.y);  // mass / density, as the record stores it
          sumker += ker * vol;
          sh = sh + sj[k] * (ker * vol);
        }
      }
    }
  } else {
    scan(celli, pos_i);
  }
  if (P.periodbound) {
    I3 cpb;
    V3<T> ppb;
    if (period_image(P, celli, pos_i, true, cpb, ppb)) scan(cpb, ppb);
  }
  if (sumker != T(0.f)) sh = sh / sumker;
  st6(S.tc_a, S.tc_b, i, sh);
}

template <class T> __global__ void k_shepard_store(const Params<T> P, DevState<T> S, const Dyn<T>* dyn,
                                                   int only_filter_steps) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int npm = dyn->npm;
  if (t >= npm) return;
  if (only_filter_steps) {
    const int st = dyn->step;
    if (!(P.stress_shepard_filter != 0 && st % P.stress_shepard_filter == 0 && st != 0)) return;
  }
  const int i = P.npb + t;
  const int c = dyn->cur_main;
  const S6<T> sh = ld6(S.tc_a, S.tc_b, i);
  st6(S.str_a[c], S.str_b[c], i, sh);
  write_rec(P, S.rec, i, S.pos[c][i], S.vel[c][i], sh, S.idm[c][i].y, S.codes[c][i].x >= 10);
}

// ---------------------------------------------------------------------------------
// Lateral wall force with FP64 accumulation (replaces the single-thread loop of
// src/utilities.cu:578-640): per-block sums in a fixed order, then one block adds
// the partial sums in block order, so the result is deterministic.
// ---------------------------------------------------------------------------------
constexpr int WF_THREADS = 256, WF_BLOCKS = 296;

// ---------------------------------------------------------------------------------
// Earth-pressure profile along the wall (cuGetValuesAlongLine, src/utilities.cu:266-322):
// three bands of thickness dr next to the wall, depth bins of size dz from z_top.  The
// reference's single loop keeps, per (band, bin), the value of the last particle in
// index order; here each particle claims its bin with atomicMax on its index and a
// second pass reads the winners' contact_mag.xx / dr, which is the same result.
// ---------------------------------------------------------------------------------
template <class T> __global__ void k_profile_claim(const Params<T> P, DevState<T> S, const Dyn<T>* dyn, double x_wall,
                                                   double z_top, double dz, int nbins, int* last) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  // The reference loops i over [npb, np): deleted particles take part too.
  if (t >= P.np - P.npb) return;
  const int i = P.npb + t;
  const int c = dyn->cur_main;
  const V4<T> ps = S.pos[c][i];
  const int4 cp = S.cellpos[c][i];
  const T h2 = (T)(2.0 * (double)P.h);
  const double px = (double)(ps.x + (T)cp.x * h2);
  const double pz = (double)(ps.z + (T)cp.z * h2);
  if (!(pz >= z_top - 1.0 && pz <= z_top)) return;
  const double dr = (double)P.dr;
  for (int band = 0; band < 3; ++band) {
    if (px >= x_wall + dr * band && px <= x_wall + dr * (band + 1)) {
      const int b = (int)((z_top - pz) / dz);
      if (b >= 0 && b < nbins) atomicMax(&last[band * nbins + b], i);
    }
  }
}

template <class T> __global__ void k_profile_read(const Params<T> P, DevState<T> S, int cpar, int nbins,
                                                  const int* last, double* out) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbins) return;
  // the depth is written with the first band's value, as the reference's .xy
  out[4 * b] = last[b] >= 0 ? (double)b * (double)P.dr : 0.0;
  for (int band = 0; band < 3; ++band) {
    const int i = last[band * nbins + b];
    out[4 * b + 1 + band] = i >= 0 ? (double)(S.cf[cpar][i].x / P.dr) : 0.0;
  }
}

template <class T> __global__ void __launch_bounds__(WF_THREADS) k_wall_force(const Params<T> P, DevState<T> S,
                                                                             const Dyn<T>* dyn, int cpar, int mode,
                                                                             int wall_id, double xmax, double zmin,
                                                                             double zmax) {
  __shared__ double red[3][WF_THREADS / 32];
  const int npm = dyn->npm, c = dyn->cur_main;
  double a[3] = {0.0, 0.0, 0.0};
  for (int t = blockIdx.x * WF_THREADS + threadIdx.x; t < npm; t += gridDim.x * WF_THREADS) {
    const int i = P.npb + t;
    bool take;
    if (mode == 0) {
      const V4<T> cv = S.cv[cpar][i];
      take = (int)cv.w == wall_id && cv.y <= P.h * T(2);
    } else {
      const V4<T> ps = S.pos[c][i];
      const int4 cp = S.cellpos[c][i];
      const double px = (double)(ps.x + (T)cp.x * (T(2.0f) * P.h));
      const double pz = (double)(ps.z + (T)cp.z * (T(2.0f) * P.h));
      take = px <= xmax && pz >= zmin && pz <= zmax;
    }
    if (take) {
      const V4<T> f = S.cf[cpar][i];
      a[0] += (double)f.x;
      a[1] += (double)f.y;
      a[2] += (double)f.z;
    }
  }
  // warp-shuffle butterfly, then the warps' partials in warp order: a fixed order, so
  // the resultant does not change from run to run
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    for (int k = 0; k < 3; ++k) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < 3; ++k) red[k][warp] = a[k];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; ++k) {
      double v = 0.0;
      for (int w = 0; w < WF_THREADS / 32; ++w) v += red[k][w];
      S.wsum[3 * blockIdx.x + k] = v;
    }
}

static __global__ void k_wall_force_final(double* wsum, int nblocks) {
  if (threadIdx.x != 0) return;
  double a[3] = {0.0, 0.0, 0.0};
  for (int b = 0; b < nblocks; ++b)
    for (int k = 0; k < 3; ++k) a[k] += wsum[3 * b + k];
  for (int k = 0; k < 3; ++k) wsum[3 * nblocks + k] = a[k];
}

// ---------------------------------------------------------------------------------
// Export of arrays whose rows are not stored as the reference lays them out: element k of a
// run of rows from `first`, written in order to the device buffer that is copied out.
// ---------------------------------------------------------------------------------
template <class T> struct Rows6 {
  const V4<T>* a;
  const V2<T>* b;
  RWD T operator()(size_t i, int k) const {
    return k < 4 ? reinterpret_cast<const T*>(a + i)[k] : reinterpret_cast<const T*>(b + i)[k - 4];
  }
};
template <class T> struct RowsContact {
  const V4<T>*f, *n, *v;
  RWD T operator()(size_t i, int k) const {
    return reinterpret_cast<const T*>((k < 3 ? f : k < 6 ? n : v) + i)[k % 3];
  }
};
struct RowsCell {
  const int2* range;
  bool end;
  RWD int operator()(size_t i, int) const {
    const int2 r = range[i];
    return r.y > r.x ? (end ? r.y : r.x) : -1;
  }
};
template <class T> struct RowsPosAbs {
  const V4<T>* pos;
  const int4* cell;
  T two_h;
  RWD T operator()(size_t i, int k) const {
    const T p = reinterpret_cast<const T*>(pos + i)[k];
    return k < 3 ? add_rn(p, rmul((T)reinterpret_cast<const int*>(cell + i)[k], two_h)) : p;
  }
};
template <class Row, class E> __global__ void k_export(Row row, size_t first, size_t n, int cols, E* out) {
  const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (k < n) out[k] = row(first + k / cols, (int)(k % cols));
}

// Totals of the kept candidate lists: out[0] += entries, out[1] += soil particles with a list.
// Per-material constants of the hypoplastic update, once per case (rw_device.cuh).
template <class T> __global__ void k_hypo_table(const Params<T> P, HypoC<T>* out) {
  const int m = threadIdx.x;
  if (m < kModelMax) out[m] = hypo_coef(P.model_par[m][0], P.model_par[m][1], P.model_par[m][2], P.model_par[m][4]);
}

static __global__ void k_list_totals(const int* cnt, int n, unsigned long long* out) {
  unsigned long long e = 0, p = 0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    if (cnt[t] >= 0) {
      e += (unsigned long long)cnt[t];
      ++p;
    }
  for (int o = 16; o > 0; o >>= 1) {
    e += __shfl_xor_sync(0xffffffffu, e, o);
    p += __shfl_xor_sync(0xffffffffu, p, o);
  }
  if ((threadIdx.x & 31) == 0 && p) {
    atomicAdd(&out[0], e);
    atomicAdd(&out[1], p);
  }
}

// ---------------------------------------------------------------------------------
// Learned constitutive closure (no counterpart in the reference): samples for its
// training and its use inside the step.  Features and target as in rw_mlp.cuh.
// ---------------------------------------------------------------------------------
struct ClosureTrust {
  float lo[mlp::IN], hi[mlp::IN];  // accepted feature ranges
  float out_max;                   // accepted |output|
  float err_max;                   // accepted judged relative error of the rate (<= 0: no bound)
};

template <class T> RWD void closure_features(const HypoPre<T>& h, const S6<T>& D, const T* mp, float* f) {
  const T ip = T(1) / h.p, inD = T(1) / h.nD;
  f[0] = (float)(h.str.xx * ip);
  f[1] = (float)(h.str.yy * ip);
  f[2] = (float)(h.str.zz * ip);
  f[3] = (float)(h.str.xy * ip);
  f[4] = (float)(h.str.xz * ip);
  f[5] = (float)(h.str.yz * ip);
  f[6] = (float)(D.xx * inD);
  f[7] = (float)(D.yy * inD);
  f[8] = (float)(D.zz * inD);
  f[9] = (float)(D.xy * inD);
  f[10] = (float)(D.xz * inD);
  f[11] = (float)(D.yz * inD);
  const T void_min = mp[9];
  f[12] = (float)((h.e - void_min) / (h.e_crt - void_min));
  f[13] = ((float)f_sin(mp[2]) - mlp::SIN_MID) / mlp::SIN_HALF;
  f[14] = (float)h.fd;  // the law's own void-ratio factor psi^alpha
  f[15] = 0.0f;
}

template <class T> RWD S6<T> closure_scale_out(const HypoPre<T>& h, const float* y) {
  const T sc = h.p * h.nD * (T)mlp::TARGET_SCALE;
  return S6<T>{(T)y[0] * sc, (T)y[1] * sc, (T)y[2] * sc, (T)y[3] * sc, (T)y[4] * sc, (T)y[5] * sc};
}

// Uniform in [0, 1) from a 64-bit key (splitmix64 finaliser).
RWD float hash_unit(unsigned long long k) {
  k += 0x9E3779B97F4A7C15ull;
  k = (k ^ (k >> 30)) * 0xBF58476D1CE4E5B9ull;
  k = (k ^ (k >> 27)) * 0x94D049BB133111EBull;
  k ^= k >> 31;
  return (float)(k >> 40) * (1.0f / 16777216.0f);
}

// Friction angle [rad] and initial void ratio ranges for augmented samples.
struct Augment {
  float phi_lo, phi_hi, e0_lo, e0_hi;
  unsigned long long seed;
  int on;
};

// Appends (features, exact normalised objective rate) of every stride-th soil particle
// with a HypoCS update, from the current stress, strain rate and density.  With
// augmentation each sample takes a friction angle and an initial void ratio drawn
// uniformly from the given ranges: the state comes from the solver, the target from the
// exact law for that material.
template <class T> __global__ void k_collect(const Params<T> P, DevState<T> S, const Dyn<T>* dyn, float* X, float* Tg,
                                             long long cap, unsigned long long* count, int stride, Augment aug) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) * stride;
  const int npm = dyn->npm, c = dyn->cur_main;
  bool ok = false;
  float f[mlp::IN], tg[mlp::OUT];
  if (t < npm) {
    const int i = P.npb + t;
    const int4 code = S.codes[c][i];
    if (code.y == 1 && code.z == RW_MODEL_HYPO_CS) {
      T mpa[kMatSize];
#pragma unroll
      for (int k = 0; k < kMatSize; ++k) mpa[k] = P.model_par[code.w][k];
      if (aug.on) {
        const unsigned long long key = aug.seed * 0x100000001B3ull + (unsigned long long)i;
        mpa[2] = (T)(aug.phi_lo + (aug.phi_hi - aug.phi_lo) * hash_unit(2 * key));
        mpa[11] = (T)(aug.e0_lo + (aug.e0_hi - aug.e0_lo) * hash_unit(2 * key + 1));
      }
      const T* mp = mpa;
      const S6<T> D = ld6(S.ace_a, S.ace_b, i);
      S6<T> sg = ld6(S.str_a[c], S.str_b[c], i);
      HypoPre<T> h;
      T mcrt;
      if (hypo_cs_pre(S.vel[c][i].w, V3<T>{T(0), T(0), T(0)}, D, sg, mp, mcrt, P.mixed != 0, h) && h.nD > T(0)) {
        closure_features(h, D, mp, f);
        const S6<T> R = hypo_cs_objective(h, D);
        const T sc = T(1) / (h.p * h.nD * (T)mlp::TARGET_SCALE);
        tg[0] = (float)(R.xx * sc);
        tg[1] = (float)(R.yy * sc);
        tg[2] = (float)(R.zz * sc);
        tg[3] = (float)(R.xy * sc);
        tg[4] = (float)(R.xz * sc);
        tg[5] = (float)(R.yz * sc);
        ok = true;
#pragma unroll
        for (int k = 0; k < mlp::IN; ++k) ok = ok && isfinite(f[k]);
#pragma unroll
        for (int o = 0; o < mlp::OUT; ++o) ok = ok && isfinite(tg[o]);
      }
    }
  }
  const unsigned mask = __ballot_sync(0xffffffffu, ok);
  if (!mask) return;
  const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(count, (unsigned long long)__popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (!ok) return;
  const long long idx = (long long)base + __popc(mask & ((1u << lane) - 1u));
  if (idx >= cap) return;
#pragma unroll
  for (int k = 0; k < mlp::IN; ++k) X[idx * mlp::IN + k] = f[k];
#pragma unroll
  for (int o = 0; o < mlp::OUT; ++o) Tg[idx * mlp::OUT + o] = tg[o];
}

// The HypoCS updates of one integrator stage (0: predictor half step, 1: corrector full
// step) with the learned objective rate: 128 soil slots per tile on the tensor cores;
// the Jaumann term, the cut-offs and every particle outside the trust region (or whose
// output leaves it) stay exact.  Every closure update is judged against the exact rate:
// stats = [offered, used, sum of relative errors, largest relative error].
// One tile of 128 soil slots; every thread of the group calls it for the same tile (the
// network runs on the whole tile).
template <class T>
RWD void closure_tile(const Params<T>& P, const DevState<T>& S, const Dyn<T>* dyn, const mlp::FwdWeights& w,
                      mlp::FwdTile& ft, int g, const ClosureTrust& tr, double* stats, int stage, int tile,
                      uint32_t& phase) {
  const int npm = dyn->npm, c = dyn->cur_main;
  const int tid = threadIdx.x & (mlp::TILE - 1), lane = tid & 31;
  const T dt = stage == 0 ? T(0.5f) * P.dt : P.dt;
  {
    const int t = tile * mlp::TILE + tid, i = P.npb + t;
    bool mine = false, act = false;
    float f[mlp::IN];
#pragma unroll
    for (int k = 0; k < mlp::IN; ++k) f[k] = 0.0f;
    int4 code{0, 0, 0, 0};
    V3<T> vs{T(0), T(0), T(0)};  // e, e_c and the void-ratio factor (two powers), kept for the update
    if (t < npm) {
      code = S.codes[c][i];
      mine = code.y == 1 && code.z == RW_MODEL_HYPO_CS;
      if (mine) {
        const T* mp = P.model_par[code.w];
        const S6<T> D = ld6(S.ace_a, S.ace_b, i);
        S6<T> sg = ld6(S.str_a[c], S.str_b[c], i);
        HypoPre<T> h;
        T mcrt;
        const HypoC<T> hc = P.hypo[code.w];
        const bool pre = hypo_cs_pre(S.vel[c][i].w, V3<T>{T(0), T(0), T(0)}, D, sg, mp, mcrt, P.mixed != 0, h, &hc);
        if (pre) vs = V3<T>{h.e, h.e_crt, h.fd};
        if (pre && h.nD > T(0)) {
          closure_features(h, D, mp, f);
          act = true;
#pragma unroll
          for (int k = 0; k < mlp::IN; ++k) act = act && f[k] >= tr.lo[k] && f[k] <= tr.hi[k];
          if (!act)
#pragma unroll
            for (int k = 0; k < mlp::IN; ++k) f[k] = 0.0f;
        }
      }
    }
    float y[mlp::OUT];
#pragma unroll
    for (int o = 0; o < mlp::OUT; ++o) y[o] = 0.0f;
    ft.any = 0;
    mlp::group_sync(g);
    if (act) ft.any = 1;
    mlp::group_sync(g);
    if (ft.any) {  // a tile without a trusted particle skips the network
      mlp::store_row<mlp::IN>(ft.h, tid, f);
      mlp::forward_tile(w, ft, g, phase, y);
    }
    float used = 0.0f, offered = 0.0f, err = 0.0f;
    if (mine) {
      const T* mp = P.model_par[code.w];
      const S6<T> D = ld6(S.ace_a, S.ace_b, i);
      const V4<T> om4 = S.spin[i];
      S6<T> sg = ld6(S.str_a[c], S.str_b[c], i);
      HypoPre<T> h;
      T mcrt = T(0);
      const HypoC<T> hc = P.hypo[code.w];
      if (hypo_cs_pre(T(0), V3<T>{om4.x, om4.y, om4.z}, D, sg, mp, mcrt, P.mixed != 0, h, &hc, &vs)) {
        S6<T> rate;
        bool use = act && !ft.err;
#pragma unroll
        for (int o = 0; o < mlp::OUT; ++o) use = use && fabsf(y[o]) <= tr.out_max;
        if (h.nD > T(0)) offered = 1.0f;
        if (use) {  // judged against the exact objective rate; kept within the error bound
          const S6<T> Rm = closure_scale_out(h, y);
          const S6<T> Rx = hypo_cs_objective(h, D);
          const S6<T> d = Rm - Rx;
          const T nx = f_sqrt(trace2(Rx, Rx)), nd = f_sqrt(trace2(d, d));
          err = (float)(nd / (nx + T(1e-30)));
          use = !(tr.err_max > 0.0f) || err <= tr.err_max;
        }
        if (use) {
          used = 1.0f;
          rate = h.jau + closure_scale_out(h, y);
        } else {
          err = 0.0f;
          rate = hypo_cs_rate(h, D);
        }
        hypo_cs_post(dt, h, rate, sg);
      }
      st6(S.str_a[c], S.str_b[c], i, sg);
      if (stage == 1) S.idm[c][i].w = mcrt;
      write_rec(P, S.rec, i, S.pos[c][i], S.vel[c][i], sg, S.idm[c][i].y, code.x >= 10);
    }
    // statistics: kept per warp until the block ends (four atomics for
    // every warp and tile queued at their one sector in L2)
    float so = offered, su = used, se = err, sx = err;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      so += __shfl_xor_sync(0xffffffffu, so, o);
      su += __shfl_xor_sync(0xffffffffu, su, o);
      se += __shfl_xor_sync(0xffffffffu, se, o);
      sx = fmaxf(sx, __shfl_xor_sync(0xffffffffu, sx, o));
    }
    if (lane == 0 && so > 0.0f) {
      stats[0] += (double)so;
      stats[1] += (double)su;
      stats[2] += (double)se;
      stats[3] = fmax(stats[3], (double)sx);
    }
  }
}

// One integrator stage (0: predictor, 1: corrector) with the learned closure, in one
// persistent launch: the rows of a tile are advanced as predictor_row / corrector_row do
// (HypoCS stresses left to the closure), then the same 128 threads run the closure on them.
// Tiles: the boundary rows first (integrator only), then the soil slots (in the predictor
// the deleted slots too, for their step-start copies).
// A tile is a chain of latencies (the rows' reads, ten barriers, five rounds of MMA, TMEM
// read and tanh), so the SM needs many: two groups of 128 threads share a block's 29 KB of
// weights and three blocks fit an SM in FP32 (80 registers, about 100 spilled bytes), 24 warps
// instead of 16.  At 223k soil particles 86 us before, 63 now: the statistics' atomics, kept
// per block now, cost 12, the third block 7, the second evaluation of the two powers 3 (four
// blocks of one tile: 70; keeping all of HypoPre across the network spills 700 bytes: 70).
// An FP64 row needs 168 registers: one tile a block, as many blocks as fit.
template <class T> constexpr int kClGroups = sizeof(T) == 4 ? 2 : 1;  // tiles a block has at a time
template <class T> constexpr int kClBlocks = sizeof(T) == 4 ? 3 : 4;  // blocks launched per SM
template <class T, int Stage>
__global__ void __launch_bounds__(mlp::TILE * kClGroups<T>, sizeof(T) == 4 ? kClBlocks<T> : 1)
    k_integrate_cl(const Params<T> P, DevState<T> S, Dyn<T>* dyn, mlp::Net net, ClosureTrust tr, double* stats) {
  constexpr int kG = kClGroups<T>;
  extern __shared__ __align__(128) unsigned char raw[];
  mlp::FwdSmem<kG>& sm = *reinterpret_cast<mlp::FwdSmem<kG>*>(raw);
  const int g = threadIdx.x / mlp::TILE, row = threadIdx.x & (mlp::TILE - 1);
  mlp::FwdTile& ft = sm.t[g];
  mlp::load_fwd(sm.w, net);
  __shared__ double warp_stats[4 * kG][4];
  double* const ws = warp_stats[threadIdx.x >> 5];
  if ((threadIdx.x & 31) < 4) ws[threadIdx.x & 31] = 0.0;
  if (row == 0) ft.err = 0;
  if (threadIdx.x == 0)
    for (int k = 1; k < kG; ++k) tc::mbar_init(&sm.t[k].bar, 1);
  mlp::block_setup(&sm.t[0].bar, &sm.w.tmem, mlp::HID * kG);
  const int nb_tiles = (P.npb + mlp::TILE - 1) / mlp::TILE;
  const int soil_rows = Stage == 0 ? P.np - P.npb : dyn->npm;
  const int n_tiles = nb_tiles + (soil_rows + mlp::TILE - 1) / mlp::TILE;
  uint32_t phase = 0;
  const RowIn<T> in = row_in<T, Stage>(S, dyn);
  for (int tile = blockIdx.x * kG + g; tile < n_tiles; tile += gridDim.x * kG) {  // group-uniform
    if (tile < nb_tiles) {
      const int i = tile * mlp::TILE + row;
      if (i < P.npb) {
        if (Stage == 0) predictor_row<false>(P, S, dyn, i, in, i);
        else corrector_row(P, S, dyn, i, in, i);
      }
      continue;
    }
    const int st = tile - nb_tiles, t = st * mlp::TILE + row;
    if (t < soil_rows) {
      if (Stage == 0) predictor_row<false>(P, S, dyn, P.npb + t, in, P.npb + t);
      else corrector_row(P, S, dyn, P.npb + t, in, P.npb + t);
    }
    closure_tile(P, S, dyn, sm.w, ft, g, tr, ws, Stage, st, phase);
  }
  mlp::group_sync(g);
  if (row == 0 && ft.err && phase > 0) tc::mbar_wait(&ft.bar, (phase - 1u) & 1u);  // MMAs of a late phase
  mlp::block_teardown(sm.w.tmem, mlp::HID * kG);
  if (threadIdx.x < 4) {  // after the barrier of the tear-down
    double v = 0.0;
    for (int k = 0; k < 4 * kG; ++k)
      v = threadIdx.x < 3 ? v + warp_stats[k][threadIdx.x] : fmax(v, warp_stats[k][3]);
    if (v != 0.0) {
      if (threadIdx.x < 3) atomicAdd(&stats[threadIdx.x], v);
      else atomicMax(reinterpret_cast<unsigned long long*>(&stats[3]), (unsigned long long)__double_as_longlong(v));
    }
  }
  if (row == 0 && ft.err) atomicOr(&dyn->err, 16u);
}

}  // namespace rw
