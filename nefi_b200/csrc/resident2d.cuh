// resident2d.cuh — many 2-D leapfrog steps per launch, the wavefield kept on the chip (sm_100a).
//
// A thread-block cluster holds one shot: CTA i of the cluster owns a slab of whole grid rows. Its two
// time levels live in shared memory (the step writes p^{n+1} over p^{n-1}, which only the owning thread
// reads), c^2 dt^2 and, in the adjoint, the gradient sums in registers. So a step moves nothing through
// L2 but Lap p (stored by the forward, read by the adjoint), the layer's coefficients and the receivers'
// samples, and costs one CTA barrier instead of a launch.
//
// Only the R rows on each side of a slab cross CTAs. The warp that computes a piece of such a row copies it
// into the halo rows of the neighbour's level over distributed shared memory (a bulk copy), which completes
// the transaction count of an mbarrier there; the threads that read the halo wait on it. A CTA therefore
// waits for its two neighbours only, and no cluster-wide barrier (with the fence it carries) is paid per
// step. p^{n+1} arrives in the halo rows that held p^{n-1}: the neighbour sends it once all of this CTA's
// edge rows of p^n have reached it, and every warp that reads a halo row of p^{n-1} sends its piece of an edge
// row of p^n after that read, so nobody reads the rows any more.
//
// Waits are bounded. A thread that gives one up waits and sends no more, its CTA arms no further phase, and the
// neighbours' waits run out in turn. The kernel runs to its end, writes NaN for all results of a shot of whose CTAs one
// gave up, and tells the host (Resident::report).
//
// Threads: a row has NV vectors of VZ = 16 / sizeof(T) columns, a slab S strips of rows; a thread steps one
// vector of one strip, marching over at most RX rows with a (2R+1)-row register window. The vectors that hold
// layer columns are the last warps' (strip by strip), the others come before them, so that few warps of a slab
// between the layers step layer cells: interleaved, 5 of the 13 warps of a 552-column slab did, and the
// others waited for them (PML 296^2, 16 shots, adjoint: 12.4 -> 10.2 us a step). The last strip marches
// upwards, so that both of a slab's edges are computed, and sent, first. One or more further warps serve the
// others: they sample the receivers, gather the next step's cotangents, arm the mbarriers. A warp without
// layer cells steps its rows without the layer's coefficients.
//
// Per-step time (fp32, order 4, one-step launches -> resident): 168^2 1 shot 3.45 -> 1.34 us forward, 2.48 -> 1.47
// adjoint; 296^2 4 shots 3.58 -> 1.99, 4.96 -> 2.29; 440^2 10 shots 6.81 -> 5.1; 552^2 16 shots 16.4 -> 13.5.
//
// The arithmetic of a cell is that of fwd2d / adj2d, operation by operation: fields and traces are
// bitwise those of the one-step launches. The gradient is summed per shot over the steps.
#pragma once
#include <climits>
#include <cmath>

#include "kernels.cuh"
#include "stencil2d.cuh"
#include "lanes.cuh"
#include "aux_kernels.cuh"

namespace nw {

constexpr int kMaxCluster = 16;

template <typename T>
struct Resident {
  typename LaneWeight<T>::t wc, w1x, w1z, w2x, w2z, minus_one;  // Laplacian weights, and -1
  // levels of the first step: forward p^{n-1}, p^n | adjoint q^{n+2}, q^{n+1}; and where the last two go
  // (nullptr, forward: nowhere)
  const T* in_prev;
  const T* in_cur;
  T* out_prev;
  T* out_cur;
  const T* C;
  const T* A;  // absorbing coefficients or nullptr
  const T* B;
  int n_first;   // first step index: the forward runs n_first, n_first + 1, ...; the adjoint downwards
  int count;     // steps
  int cluster;   // CTAs per shot
  int nv;        // vectors per row
  int strips;    // strips per slab
  int max_rows;  // rows of the largest slab
  // PML: coefficients, the face fields of the first step (x, z faces) and where the last ones go
  const T* zz;
  const T* alpha[2];
  const T* beta[2];
  const T* f_in[2];
  T* f_out[2];
  T hx2, hz2;  // 0.5 / h
  int core_x0, core_x1;  // rows without layer cells between the edge columns
  int edge_lo, edge_hi;  // vectors [0, edge_lo) and [edge_hi, nv) hold layer columns
  int slab[kMaxCluster + 1];  // first row of each CTA's slab
  int substeps, first_b_one;
  long long level;  // elements of one level (Lap p levels are consecutive)
  // forward
  const int* __restrict__ src_corner;
  const T* __restrict__ src_w;
  const T* __restrict__ wavelet;
  T* traces;  // nullptr: no samples
  const int* __restrict__ rec_corner;
  const T* __restrict__ rec_w;
  T* lap_out;  // Lap p of step n_first (step n at + (n - n_first) levels), or nullptr
  T* snap;     // exact snapshots: the levels p^{n-1}, p^n (with a PML the face fields, too) of every step n that
               // is a multiple of `segment` go to snap + (n / segment) * snap_stride; nullptr: none
  int segment;
  long long snap_stride;
  // adjoint
  const T* __restrict__ gtr;  // trace cotangents, or nullptr
  const int64_t* __restrict__ cell_index;
  const int* __restrict__ cell_ptr;
  const int* __restrict__ cell_rec;
  const T* __restrict__ cell_w;
  const T* __restrict__ lap;  // Lap p of step 0 in memory order (step n at + (n - lap_n0) levels)
  int lap_n0, lap_end;        // steps [lap_n0, lap_end) have a Lap p; others add nothing to the gradient
  T* acc;                     // per-shot sums of q^{n+1} Lap p^n (read, added to, written)
  // forward of a time reversal: after step n the imposed cells (field offsets, n_imposed) hold their traces at
  // reversed time T - (n + 1) dt, linear between samples
  const int64_t* __restrict__ imposed;
  const T* __restrict__ imposed_tr;
  int n_imposed;
  int n_rec, n_t, n_cells;
  int mute;        // 1: the first CTA of a shot sends nothing (to test what follows)
  int* report;     // host memory: set to NW_ERR_TIMEOUT when a wait gave up
  int cap_list;  // receivers (forward) or touched cells (adjoint) the shared tables hold: at least all of them
  int cap_ent;   // adjoint: the table entries they hold
};

// Threads per CTA at most: 16 warps leave each 128 registers, which hold c^2 dt^2 and, in the adjoint, the
// gradient sums of RX vectors beside the 2R+1-row window (more warps would spill them).
// A PML's strips hold more beside them: 12 warps of 168 registers.
__host__ __device__ constexpr int resident_threads(bool pml) { return pml ? 384 : 512; }

// Threads that step cells: the vectors without layer columns of all strips, then the others, each rounded up to
// warps.
__host__ __device__ inline int resident_cell_threads(int nv, int edge_lo, int edge_hi, int strips) {
  const int n_in = edge_hi - edge_lo;
  return (strips * n_in + 31) / 32 * 32 + (strips * (nv - n_in) + 31) / 32 * 32;
}

// Shared memory: two levels of the slab with R halo rows above and below (a zero vector before the first
// row and after each row), the mbarriers, then the tables.
template <typename T, int R>
struct ResidentSmem {
  static constexpr int VZ = 16 / (int)sizeof(T);
  __host__ __device__ static int pitch(int nv) { return (nv + 1) * VZ; }
  __host__ __device__ static int level(int nv, int rows) { return VZ + (rows + 2 * R) * pitch(nv); }
  __host__ __device__ static size_t tables(int nv, int rows, int levels) {  // byte offset of the tables
    return levels * (size_t)level(nv, rows) * sizeof(T) + 4 * 8 + 16;
  }
  static constexpr size_t list_entry = 8 + 4 * sizeof(T);                 // forward: id, offset, 4 weights
  static constexpr size_t cell_entry = 4 + 2 * sizeof(T);                 // adjoint: first entry, 2 values
  static constexpr size_t csr_entry = 4 + sizeof(T);                      // offset, weight
  static constexpr size_t imposed_entry = 4 + 2 * sizeof(T);              // trace, 2 values
  __host__ __device__ static size_t lane_bytes(int nv, int rows) { return ((size_t)nv * rows * VZ * 2 + 15) / 16 * 16; }
  __host__ __device__ static size_t map_bytes(int nv, int rows) { return ((size_t)nv * rows * 2 + 15) / 16 * 16; }
  // A, B: one vector each per row (its columns between the layers, all alike), those of the edge vectors
  __host__ __device__ static size_t coef_bytes(int ne, int rows) { return (size_t)rows * (ne + 1) * 32; }
  // PML: seven coefficient fields over the rows and the first one below, likewise (two more edge vectors: the
  // faces after each edge), and the face fields: x faces, z faces by step parity
  static constexpr int kPmlCo = 7;
  __host__ __device__ static size_t pml_bytes(int ne, int nv, int rows) {
    return (size_t)kPmlCo * (rows + 1) * (ne + 3) * 16 + (size_t)3 * rows * pitch(nv) * sizeof(T);
  }
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// Address of this CTA's shared-memory location `a` in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned map_cta(unsigned a, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// The CTA's barrier from different places of the code (warp-uniform).
__device__ __forceinline__ void cta_barrier() { asm volatile("barrier.sync 0;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of parity `par`; false if it did not complete within 2^17 tries, 0.2 s. (A try that fails takes
// 1.5 us, measured. A limit that is no constant, or a look at the clock, cost a step of 128^2 or 256^2 0.2 to 0.6 us.)
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned par) {
  for (int i = 0; i < (1 << 17); ++i) {
    unsigned done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(par)
        : "memory");
    if (done) return true;
  }
  return false;
}
// `bytes` from this CTA's shared memory to a cluster address, completing as many bytes of the transaction
// count of `bar` (in the destination's CTA). The copy reads through the async proxy: the writers fence first.
__device__ __forceinline__ void send_bytes(unsigned dst, unsigned src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "r"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// The Laplacian of the window's centre row, lane by lane the operations of lap_at (the terms of the two
// neighbours along an axis commute, so a march upwards gives the same bits).
template <typename T, int R, int VZ>
__device__ __forceinline__ void lap_row(const T (&wv)[2 * R + 1][VZ], const Row3<T, VZ>& rw, const Resident<T>& a,
                                        T (&lap)[VZ]) {
  T t[VZ];
  v_mul(a.wc, wv[R], lap);
  v_add(wv[R - 1], wv[R + 1], t);
  v_fma(a.w1x, t, lap, lap);
#pragma unroll
  for (int v = 0; v < VZ; ++v) t[v] = add_rn(zval(rw, v - 1), zval(rw, v + 1));
  v_fma(a.w1z, t, lap, lap);
  if constexpr (R == 2) {
    v_add(wv[0], wv[4], t);
    v_fma(a.w2x, t, lap, lap);
    T zl[VZ], zr[VZ];
#pragma unroll
    for (int v = 0; v < VZ; ++v) {
      zl[v] = zval(rw, v - 2);
      zr[v] = zval(rw, v + 2);
    }
    v_add(zl, zr, t);
    v_fma(a.w2z, t, lap, lap);
  }
}

// Numbers of elements of the ascending list `idx` below two bounds, counted by the whole CTA.
__device__ __forceinline__ int2 count_below(const int64_t* idx, int n, long long b0, long long b1) {
  int2 total = make_int2(0, 0);
  for (int b = 0; b < n; b += blockDim.x) {
    const int i = b + threadIdx.x;
    const int64_t v = i < n ? idx[i] : b1;
    total.x += __syncthreads_count(v < b0);
    total.y += __syncthreads_count(v < b1);
  }
  return total;
}

// The report to the host, and NaN in the place of all that a CTA of shot s has written: in the levels, the gradient sums, Lap p and the snapshots the
// strip of `nr` rows whose first vector (of column zc) is at `cell`, and all samples. Copies that nobody waited for then
// have had a millisecond to land. (Not inlined: it would cost the time loops registers.)
template <typename T, int VZ, bool ADJ>
__device__ __noinline__ void mark_lost(const Resident<T>& a, int s, long long cell, int nr, int dld, int zc, int n1) {
  const long long t0 = clock64();
  *(volatile int*)a.report = 5;  // NW_ERR_TIMEOUT
  T bad[VZ];
  for (int v = 0; v < VZ; ++v) bad[v] = T(NAN);
  for (int k = 0; k < nr; ++k, cell += dld) {
    T* fields[3] = {a.out_cur, a.out_prev, ADJ ? a.acc : nullptr};
    for (T* f : fields)
      if (f) store_row<T, VZ>(f + cell, bad, zc, n1);
    for (int n = a.n_first; !ADJ && n < a.n_first + a.count; ++n) {
      if (a.lap_out) store_row<T, VZ>(a.lap_out + (n - a.n_first) * a.level + cell, bad, zc, n1);
      if (a.snap && n % a.segment == 0)
        for (int l = 0; l < 2; ++l)
          store_row<T, VZ>(a.snap + (long long)(n / a.segment) * a.snap_stride + l * a.level + cell, bad, zc, n1);
    }
  }
  if (!ADJ && a.traces)
    for (int n = a.n_first; n < a.n_first + a.count; ++n)
      for (int e = threadIdx.x; n % a.substeps == 0 && e < a.n_rec; e += blockDim.x)
        a.traces[((long long)s * a.n_rec + e) * a.n_t + n / a.substeps] = T(NAN);
  for (int i = 0; i < 10000 && clock64() - t0 < 2000000; ++i) __nanosleep(1000);
}

// IMP: the forward of a time reversal, which imposes cells after each step (apart: it costs registers).
template <typename T, int R, int RX, bool ADJ, bool PML, bool IMP>
__global__ void __launch_bounds__(resident_threads(PML), 1) resident2d(const __grid_constant__ KGrid<T> g, const __grid_constant__ Resident<T> a) {
  using L = ResidentSmem<T, R>;
  constexpr int VZ = L::VZ;
  constexpr int PF = RX > 6 ? 1 : 2;  // rows of Lap p loaded ahead (adjoint)
  // the adjoint of the tallest strips has no registers left for c^2 dt^2: it streams it from L2
  constexpr bool C_REG = !(ADJ && RX > 6);
  // The step overwrites the older level, except with a PML's adjoint, whose face fields read it at the
  // neighbours too
  constexpr int NL = PML && ADJ ? 3 : 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int rank = (int)cluster_rank(), s = blockIdx.x / a.cluster;
  const int X0 = a.slab[rank], rows = a.slab[rank + 1] - X0;
  const int nthr = blockDim.x, tid = threadIdx.x;
  const int pitch = L::pitch(a.nv), BS = L::level(a.nv, a.max_rows);
  T* buf = reinterpret_cast<T*>(smem_raw) + VZ;  // level b at buf + b * BS, row r (-R .. rows + R - 1) at + (r + R) * pitch
  unsigned long long* mbar = reinterpret_cast<unsigned long long*>(smem_raw + NL * (size_t)BS * sizeof(T));  // [side][2]
  int* count = reinterpret_cast<int*>(mbar + 4);
  unsigned char* tables = smem_raw + L::tables(a.nv, a.max_rows, NL);
  const unsigned mbar_a = smem_addr(mbar);
  const bool has_up = rank > 0, has_dn = rank + 1 < a.cluster;

  // ---- this thread's strip
  const int svc = resident_cell_threads(a.nv, a.edge_lo, a.edge_hi, a.strips);  // first service thread
  const int n_in = a.edge_hi - a.edge_lo, in_thr = (a.strips * n_in + 31) / 32 * 32, n_edge_vec = a.nv - n_in;
  const bool edge_thr = tid >= in_thr;
  const int strip = edge_thr ? (tid - in_thr) / max(n_edge_vec, 1) : tid / max(n_in, 1);
  const int in_group = edge_thr ? tid - in_thr - strip * n_edge_vec : tid - strip * n_in;
  const int vec = !edge_thr ? a.edge_lo + in_group : in_group < a.edge_lo ? in_group : in_group - a.edge_lo + a.edge_hi;
  const bool work = tid < svc && strip < a.strips;
  const int ra = work ? rows * strip / a.strips : 0;
  const int rb = work ? rows * (strip + 1) / a.strips : 0;
  const int nr = rb - ra;                                 // rows of the strip (<= RX)
  const bool up = !PML && a.strips > 1 && strip == a.strips - 1;  // marches from its last row upwards
  const int r0 = up ? rb - 1 : ra, dir = up ? -1 : 1;     // row of step k of the march: r0 + dir * k
  const int zc = vec * VZ;
  const int ld = (int)g.s0;
  const long long so = (long long)s * g.field;
  const int cell0 = (int)g.origin + (X0 + r0) * ld + zc;  // field offset of the march's first vector
  const int dld = dir * ld, dp = dir * pitch, po0 = (R + r0) * pitch + zc;


  // ---- shared memory: zeros, the tables' counters, the mbarriers
  T zero[VZ];
#pragma unroll
  for (int u = 0; u < VZ; ++u) zero[u] = T(0);
  for (int i = tid; i < NL * (BS / VZ); i += nthr) vstore<T, VZ>(buf - VZ + i * VZ, zero);
  __shared__ int gave_up, lost_sh;  // a wait of this CTA, of one of the shot's CTAs, gave up
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(mbar_a + 8 * i);
    count[0] = 0;
    gave_up = lost_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  // levels: own rows of both, halo rows of the current one (with three levels, of both)
  auto in_grid = [&](T (&c)[VZ], int n) {  // zeros past column n
#pragma unroll
    for (int u = 0; u < VZ; ++u)
      if (zc + u >= n) c[u] = T(0);
  };
  if (work) {
    const int h_up = has_up ? R : 0, h_dn = has_dn ? R : 0;
#pragma unroll 2
    for (int r = strip - h_up; r < rows + h_dn; r += a.strips) {
      const long long o = so + g.origin + (X0 + r) * ld + zc;
      T* dst = buf + (r + R) * pitch + zc;
      T c[VZ], p[VZ];
      vload<T, VZ>(a.in_cur + o, c);
      vload<T, VZ>(a.in_prev + o, p);
      in_grid(c, g.n1);
      in_grid(p, g.n1);
      vstore<T, VZ>(dst, c);
      // (the level that step 0 reads as the older one)
      if (NL == 3 || (r >= 0 && r < rows)) vstore<T, VZ>(dst + (NL - 1) * BS, p);
    }
  }
  // registers: c^2 dt^2, the gradient sums
  T cc[C_REG ? RX : PF][VZ], gs[ADJ ? RX : 1][VZ];
#pragma unroll
  for (int k = 0; k < RX; ++k) {
    if (k < (C_REG ? RX : PF)) {
#pragma unroll
      for (int v = 0; v < VZ; ++v) cc[k][v] = T(0);
      if (k < nr) vldg<T, VZ>(a.C + cell0 + k * dld, cc[k]);
    }
    if constexpr (ADJ) {
#pragma unroll
      for (int v = 0; v < VZ; ++v) gs[k][v] = T(0);
      if (a.acc && k < nr) vload<T, VZ>(a.acc + so + cell0 + k * dld, gs[k]);
    }
  }
  // A and B of the layer: the coefficients of a row between the edge columns are one pair (checked; the
  // layers' profiles depend on the depth below the nearest side there), those of the edge columns vectors
  const int ne = a.edge_lo + (a.nv - a.edge_hi);
  T* co_edge = reinterpret_cast<T*>(tables);                  // [A | B][rows][ne][VZ]
  T* co_row = co_edge + (size_t)2 * a.max_rows * ne * VZ;     // [A | B][rows][VZ]
  bool alike = true;
  T *pml_row = nullptr, *psi0 = nullptr, *psi1 = nullptr;  // PML: see below
  if constexpr (PML) {
    // [field][row, one more][edge vectors, the vector after each edge, the row's vector][VZ]
    const T* src[L::kPmlCo] = {a.A, a.B, a.zz, a.alpha[0], a.beta[0], a.alpha[1], a.beta[1]};
    const int w = ne + 3;
    pml_row = reinterpret_cast<T*>(tables);
    psi0 = pml_row + (size_t)L::kPmlCo * (a.max_rows + 1) * w * VZ;
    psi1 = psi0 + (size_t)a.max_rows * pitch;
    tables += L::pml_bytes(ne, a.nv, a.max_rows);
    for (int i = tid; i < 3 * a.max_rows * (pitch / VZ); i += nthr) vstore<T, VZ>(psi0 + i * VZ, zero);
    const int fs = (a.max_rows + 1) * w * VZ;
    auto take = [&](int r, int v) {  // the coefficients of vector v of row r
      const int o = (int)g.origin + (X0 + r) * ld;
      const bool inner = v >= a.edge_lo && v < a.edge_hi;
      T c[L::kPmlCo][VZ], c0[L::kPmlCo];
#pragma unroll
      for (int f = 0; f < L::kPmlCo; ++f) {
#pragma unroll
        for (int u = 0; u < VZ; ++u) c[f][u] = T(0);
        c0[f] = T(0);
        if (v * VZ < ld) vldg<T, VZ>(src[f] + o + v * VZ, c[f]);  // (vector nv, past the grid, may lie past the row)
        if (inner) c0[f] = src[f][o + a.edge_lo * VZ];
      }
#pragma unroll
      for (int f = 0; f < L::kPmlCo; ++f) {
        T* dst = pml_row + f * fs + r * w * VZ;
        if (v <= a.edge_lo) vstore<T, VZ>(dst + v * VZ, c[f]);
        if (v >= a.edge_hi) vstore<T, VZ>(dst + (v - a.edge_hi + a.edge_lo + 1) * VZ, c[f]);
        if (inner) {
#pragma unroll
          for (int u = 0; u < VZ; ++u) alike = alike && c[f][u] == c0[f];
          if (v == a.edge_lo) vstore<T, VZ>(dst + (w - 1) * VZ, c[f]);
          if (v + 1 == a.edge_hi && f >= 5) alike = alike && src[f][o + a.edge_hi * VZ] == c0[f];
        }
      }
    };
    if (work)
      for (int r = strip; r <= rows; r += a.strips) {
        take(r, vec);
        if (vec == a.nv - 1) take(r, a.nv);
      }
    alike = __syncthreads_and(alike);
    if (work)
#pragma unroll 2
      for (int r = strip; r < rows; r += a.strips) {
        const long long o = so + g.origin + (X0 + r) * ld + zc;
        T c[VZ], p[VZ];
        vload<T, VZ>(a.f_in[0] + o, c);
        vload<T, VZ>(a.f_in[1] + o, p);
        in_grid(c, g.n1);
        in_grid(p, g.n1 + 1);
        vstore<T, VZ>(psi0 + r * pitch + zc, c);
        vstore<T, VZ>(psi1 + r * pitch + zc, p);
        if (zc + VZ == g.n1) psi1[r * pitch + g.n1] = a.f_in[1][o + VZ];
      }
  } else if (a.A) {
    tables += L::coef_bytes(ne, a.max_rows);
    if (work)
#pragma unroll 2
      for (int r = strip; r < rows; r += a.strips) {
        const int o0 = (int)g.origin + (X0 + r) * ld;
        T ca[VZ], cb[VZ];
        vldg<T, VZ>(a.A + o0 + zc, ca);
        vldg<T, VZ>(a.B + o0 + zc, cb);
        if (vec < a.edge_lo || vec >= a.edge_hi) {
          T* e = co_edge + (r * ne + (vec < a.edge_lo ? vec : vec - a.edge_hi + a.edge_lo)) * VZ;
          vstore<T, VZ>(e, ca);
          vstore<T, VZ>(e + a.max_rows * ne * VZ, cb);
        } else {
          const T a0 = a.A[o0 + a.edge_lo * VZ], b0 = a.B[o0 + a.edge_lo * VZ];
#pragma unroll
          for (int u = 0; u < VZ; ++u) alike = alike && ca[u] == a0 && cb[u] == b0;
          if (vec == a.edge_lo) {
            vstore<T, VZ>(co_row + VZ * r, ca);
            vstore<T, VZ>(co_row + VZ * (a.max_rows + r), cb);
          }
        }
      }
    alike = __syncthreads_and(alike);
  }
  // where this thread's coefficients of the march's first row are, and the step to the next row's: shared
  // memory, or the field itself when the rows are not alike
  const bool edge_vec = vec < a.edge_lo || vec >= a.edge_hi;
  const int co_pitch = (edge_vec ? ne : 1) * VZ;
  const T* co_a = edge_vec ? co_edge + (vec < a.edge_lo ? vec : vec - a.edge_hi + a.edge_lo) * VZ : co_row;
  const T* co_b = co_a + a.max_rows * co_pitch;
  co_a += r0 * co_pitch;
  co_b += r0 * co_pitch;
  int co_d = dir * co_pitch;
  if (!PML && a.A && !alike) {
    co_a = a.A + cell0;
    co_b = a.B + cell0;
    co_d = dld;
  }
  // a warp steps its rows with the layer's coefficients if any of its cells lies in the layer
  const bool layer_warp =
      __any_sync(0xffffffffu, work && a.A && (edge_vec || X0 + ra < a.core_x0 || X0 + rb > a.core_x1));
  // the march's first R rows are the slab's edge (the last strip's, marching up, too); with one strip, its
  // last R rows are the lower edge
  const bool send_up = work && strip == 0 && has_up, send_dn = work && up && has_dn,
             send_late = work && strip == a.strips - 1 && !up && has_dn;
  unsigned rare = 0;  // rows of the march with the shot's source (forward) or touched cells (adjoint)

  // ---- tables: the slab's receivers (forward), the slab's touched cells and their entries (adjoint)
  int* l_id = reinterpret_cast<int*>(tables);  // forward: offset of the samples, level offset of the corner, weights
  int* l_off = l_id + a.cap_list;
  T* l_w = reinterpret_cast<T*>(l_off + a.cap_list);
  unsigned short* map = reinterpret_cast<unsigned short*>(tables);  // adjoint: per vector (first cell << 4 | lanes)
  T* c_val = reinterpret_cast<T*>(tables + L::map_bytes(a.nv, a.max_rows));  // [2][cap_list] cotangents by step parity
  T* e_w = c_val + 2 * a.cap_list;                           // [cap_ent] weights of the entries
  int* c_first = reinterpret_cast<int*>(e_w + a.cap_ent);    // [cap_list] a cell's first entry
  int* e_off = c_first + a.cap_list;                         // [cap_ent] receiver * n_t
  // count[0], count[1]: receivers inside the slab, and those that also read the halo below (at the list's
  // end); touched cells and entries
  unsigned short* lane_map = reinterpret_cast<unsigned short*>(tables);  // time reversal: a cell's entry + 1
  T* i_val = reinterpret_cast<T*>(tables + L::lane_bytes(a.nv, a.max_rows));  // [2][n_imposed] values by step parity
  int* i_row = reinterpret_cast<int*>(i_val + 2 * a.n_imposed);               // trace row
  auto imposed_values = [&](int n, T* dst, int id, int step) {  // of level n
    const double u = (a.n_t - 1) - (double)n / a.substeps;
    const int j0 = min(max((int)floor(u), 0), a.n_t - 1), j1 = min(j0 + 1, a.n_t - 1);
    const double w = u - j0;
    for (int e = id, n_in = count[0]; e < n_in; e += step) {
      const T* tr = a.imposed_tr + (long long)i_row[e] * a.n_t;
      dst[e] = add_rn(mul_rn((T)(1.0 - w), tr[j0]), mul_rn((T)w, tr[j1]));
    }
  };
  if constexpr (!ADJ) {
    if constexpr (IMP) {
      for (int i = tid; i < a.nv * rows * VZ; i += nthr) lane_map[i] = 0;
      __syncthreads();
      for (int c = tid; c < a.n_imposed; c += nthr) {
        const int rel = (int)(a.imposed[c] - g.origin) - X0 * ld;
        if (rel < 0 || rel >= rows * ld) continue;
        const int e = atomicAdd(count, 1), r = rel / ld;
        i_row[e] = c;
        lane_map[r * a.nv * VZ + rel - r * ld] = (unsigned short)(e + 1);
      }
      __syncthreads();
      imposed_values(a.n_first + 1, i_val, tid, nthr);
      if (work)
        for (int k = 0; k < nr; ++k)
#pragma unroll
          for (int v = 0; v < VZ; ++v)
            if (lane_map[(r0 + dir * k) * a.nv * VZ + zc + v]) rare |= 1u << k;
    }
    if (a.traces) {
      if (tid == 0) count[1] = 0;
      __syncthreads();
      for (int r = tid; r < a.n_rec; r += nthr) {
        const int x = a.rec_corner[2 * r] - X0, z = a.rec_corner[2 * r + 1];
        if (x < 0 || x >= rows) continue;
        const int e = x + 1 < rows ? atomicAdd(count, 1) : a.cap_list - 1 - atomicAdd(count + 1, 1);
        l_id[e] = r * a.n_t;
        l_off[e] = (x + R) * pitch + z;
#pragma unroll
        for (int k = 0; k < 4; ++k) l_w[4 * e + k] = a.rec_w[4 * r + k];
      }
    }
  } else if (a.gtr && a.n_cells > 0) {
    const int2 range = count_below(a.cell_index, a.n_cells, g.origin + (long long)X0 * ld,
                                   g.origin + (long long)(X0 + rows) * ld);
    const int eb = range.x, ee = range.y;
    const int q0 = a.cell_ptr[eb], n_ent = a.cell_ptr[ee] - q0;
    if (tid == 0) { count[0] = ee - eb; count[1] = n_ent; }
    for (int i = tid; i < a.nv * rows; i += nthr) map[i] = 0;
    __syncthreads();
    auto vec_of = [&](int e) {  // the slab vector a cell lies in, its lane in the low bits
      const int rel = (int)(a.cell_index[e] - g.origin) - X0 * ld;
      const int r = rel / ld, z = rel - r * ld;
      return (r * a.nv + z / VZ) * VZ + z % VZ;
    };
    for (int e = eb + tid; e < ee; e += nthr) {
      const int w = vec_of(e);
      c_first[e - eb] = a.cell_ptr[e] - q0;
      if (e > eb && vec_of(e - 1) / VZ == w / VZ) continue;  // the vector's first cell writes its entry
      unsigned m = 1u << (w % VZ);
      for (int f = e + 1; f < ee && f < e + VZ; ++f) {
        const int w2 = vec_of(f);
        if (w2 / VZ != w / VZ) break;
        m |= 1u << (w2 % VZ);
      }
      map[w / VZ] = (unsigned short)((e - eb) << 4 | m);
    }
    for (int q = tid; q < n_ent; q += nthr) {
      e_w[q] = a.cell_w[q0 + q];
      e_off[q] = a.cell_rec[q0 + q] * a.n_t;
    }
    __syncthreads();
    if (work)
#pragma unroll
      for (int k = 0; k < RX; ++k)
        if (k < nr && map[(r0 + dir * k) * a.nv + vec]) rare |= 1u << k;
  }
  const bool inject = ADJ && a.gtr && a.n_cells > 0;
  // the cotangents of sample j at the slab's touched cells, summed in table order, by n threads
  auto cotangents = [&](int j, T* dst, int id, int n) {
    const T* src = a.gtr + (long long)s * a.n_rec * a.n_t + j;
    const int n_list = count[0], n_ent = count[1];
#pragma unroll 2
    for (int e = id; e < n_list; e += n) {
      const int q0 = c_first[e], q1 = e + 1 < n_list ? c_first[e + 1] : n_ent;
      T v = T(0);
#pragma unroll 4
      for (int q = q0; q < q1; ++q) v = fma_rn(e_w[q], __ldg(src + e_off[q]), v);
      dst[e] = v;
    }
  };
  // sample (forward) or cotangent (adjoint) index of the step, and steps since it
  int j = a.n_first / a.substeps, phase = a.n_first - j * a.substeps;
  if (ADJ && inject && phase == 0) cotangents(j, c_val, tid, nthr);

  // ---- the source stencil of this shot (forward): the rows of the march it touches in this vector
  __shared__ T src_sh[8];  // by step parity: weights times the step's wavelet value
  if constexpr (!ADJ) {
    if (a.src_corner) {
      const int bx = a.src_corner[2 * s] - X0, bz = a.src_corner[2 * s + 1];
      if (work && bz + 1 >= zc && bz < zc + VZ) {
#pragma unroll
        for (int k = 0; k < RX; ++k)
          if (k < nr && (unsigned)(r0 + dir * k - bx) <= 1u) rare |= 1u << k;
      }
      if (tid < 4) src_sh[tid] = mul_rn(a.src_w[4 * s + tid], a.wavelet[a.n_first]);
    }
  }
  T f_end[VZ];  // PML: the x faces below the strip, which it advances on its own like the strip below does
#pragma unroll
  for (int v = 0; v < VZ; ++v) f_end[v] = T(0);
  if constexpr (PML) {
    if (work) vload<T, VZ>(a.f_in[0] + so + cell0 + (long long)nr * ld, f_end);
  }
  const bool need_up = work && has_up && ra - R < 0, need_dn = work && has_dn && rb + R > rows;
  bool dead = false;  // a wait of this thread gave up: it runs on without waiting or sending
  // (The results are marked at the end: NaN put into the rows or registers here cost a step of 128^2 3 % and more.)
  auto give_up = [&]() {
    dead = true;
    *(volatile int*)&gave_up = 1;
  };
  auto wait_halo = [&](int side, int m) {
    if (m == 0 || dead) return;
    if (!mbar_wait(mbar_a + 16 * side + 8 * (m & 1), ((m - 1) >> 1) & 1)) give_up();
  };
  T lpb[PF][VZ];  // Lap p of the next rows (adjoint)
  auto lap_of = [&](int n) -> const T* {  // this march's Lap p of step n
    return n >= a.lap_n0 && n < a.lap_end ? a.lap + (long long)(n - a.lap_n0) * a.level + so + cell0 : nullptr;
  };
  const T* lap_now = nullptr;
  if constexpr (ADJ) {
    if (work) lap_now = lap_of(a.n_first);
#pragma unroll
    for (int k = 0; k < PF && k < RX; ++k)
      if (lap_now && k < nr) vldcg<T, VZ>(lap_now + k * dld, lpb[k]);
  }
  // R edge rows of this thread's vector's piece (the lanes of this warp with adjoining vectors of the same strip:
  // one piece of a row, sent by its first lane) of the new level into the halo rows of the CTA above (side 0) or below. A shared
  // address of this CTA and the same one of a neighbour differ by a constant; row r of this slab is row r + R of
  // theirs below the slab above's last one, and row r - (rows - R) of the slab below.
  const unsigned up_off = has_up ? map_cta(mbar_a, rank - 1) - mbar_a : 0, dn_off = has_dn ? map_cta(mbar_a, rank + 1) - mbar_a : 0;
  const int run_lo = !edge_thr ? a.edge_lo : vec < a.edge_lo ? 0 : a.edge_hi, run_hi = !edge_thr ? a.edge_hi : vec < a.edge_lo ? a.edge_lo : a.nv;
  __shared__ unsigned short seg_sh[resident_threads(PML)];  // first and end lane of a thread's piece
  seg_sh[tid] = (unsigned short)(max(0, (tid & 31) - (vec - run_lo)) | min(32, (tid & 31) + run_hi - vec) << 8);
  __syncthreads();
  auto send_rows = [&](int side, bool upwards, int m, int level) {
    const int seg = seg_sh[threadIdx.x], seg_first = seg & 255, seg_end = seg >> 8;
    const unsigned mask = (seg_end == 32 ? ~0u : (1u << seg_end) - 1) & ~((1u << seg_first) - 1);
    fence_async();
    __syncwarp(mask);
    if (((int)threadIdx.x & 31) != seg_first || dead) return;
    const int row_b = pitch * (int)sizeof(T);
    const unsigned own = smem_addr(buf) + zc * (unsigned)sizeof(T) + level * (unsigned)(BS * (int)sizeof(T));
    const unsigned to = own + (side ? dn_off + (R - rows) * row_b : up_off + (R + X0 - a.slab[rank - 1]) * row_b);
    const unsigned bar = mbar_a + (side ? dn_off : up_off + 16) + 8 * ((m + 1) & 1);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = side ? (upwards ? rows - 1 - i : rows - R + i) : i;
      send_bytes(to + r * row_b, own + (r + R) * row_b, (seg_end - seg_first) * 16, bar);
    }
  };
  // The service warps' piece of a send: a zero vector into the pad of the first halo row of the CTA below.
  // It releases the bottom halo rows only after the receivers that read them are sampled.
  const bool sampled = !ADJ && a.traces != nullptr;
  cluster_barrier();  // every level read, every mbarrier initialised
  if (a.mute && rank == 0 && (need_dn || (tid >= svc && has_dn))) give_up();

  // The shot's source onto a vector of slab row r.
  auto add_source = [&](int r, int m, T (&o)[VZ]) {
    const int dx = r + X0 - a.src_corner[2 * s], z0 = zc - a.src_corner[2 * s + 1];
    const T* w = src_sh + 4 * (m & 1) + 2 * dx;
#pragma unroll
    for (int v = 0; v < VZ; ++v)
      if ((unsigned)(z0 + v) <= 1u) o[v] = add_rn(o[v], w[z0 + v]);
  };
  // Whether the edge rows may be sent as soon as they are marched over: not where cells are still to change
  // after the march, the source of a warp without the layer or a time reversal's cells, in this or another
  // thread of the piece.
  const bool early = ADJ || (!IMP && __all_sync(0xffffffffu, rare == 0));
  // Time reversal: the imposed cells of this strip's new level, before its edge rows are sent.
  auto impose = [&](int m, int level) {
    for (unsigned left = rare; left; left &= left - 1) {
      const int r = r0 + dir * (__ffs(left) - 1);
      T* row = buf + level * BS + (R + r) * pitch + zc;
#pragma unroll
      for (int v = 0; v < VZ; ++v) {
        const int e = lane_map[r * a.nv * VZ + zc + v];
        if (e) row[v] = i_val[(m & 1) * a.n_imposed + e - 1];
      }
    }
  };
  // This strip's rows of p^{n-1}, p^n and the face fields before step m, to the snapshot of step n.
  auto snapshot = [&](int m, int n) {
    T* dst = a.snap + (long long)(n / a.segment) * a.snap_stride + so + cell0;
    const T *c = buf + (m % NL) * BS + po0, *p = buf + ((m + NL - 1) % NL) * BS + po0;
    for (int k = 0; k < nr; ++k) {
      const int o = k * dld;
      T v0[VZ];
      vload<T, VZ>(p + k * dp, v0);
      store_row<T, VZ>(dst + o, v0, zc, g.n1);
      vload<T, VZ>(c + k * dp, v0);
      store_row<T, VZ>(dst + a.level + o, v0, zc, g.n1);
      if constexpr (PML) {
        vload<T, VZ>(psi0 + (r0 + k) * pitch + zc, v0);
        store_row<T, VZ>(dst + 2 * a.level + o, v0, zc, g.n1);
        const T* f1 = psi1 + ((m & 1) * a.max_rows + r0 + k) * pitch + zc;
        vload<T, VZ>(f1, v0);
        store_row<T, VZ>(dst + 3 * a.level + o, v0, zc, g.n1 + 1);
        if (zc + VZ == g.n1) dst[3 * a.level + o + VZ] = f1[VZ];
      }
    }
    if constexpr (PML) {
      if (X0 + rb == g.n0) store_row<T, VZ>(dst + 2 * a.level + nr * ld, f_end, zc, g.n1);
    }
  };
  // steps until the next snapshot (0: this one)
  const int snap0 = !ADJ && a.snap ? (a.segment - a.n_first % a.segment) % a.segment : INT_MAX;

  // The steps of this thread's strip; LAYER: with the layer's coefficients. (The time loops of the three kinds
  // of warp are apart, so that each keeps only its own values in registers.)
  auto steps = [&](auto layer_tag) {
    constexpr bool LAYER = decltype(layer_tag)::value;
    T* lpo = !ADJ && a.lap_out ? a.lap_out + so + cell0 : nullptr;
    int phase_c = phase, to_snap = snap0;
    for (int m = 0; m < a.count; ++m) {
      const int n = ADJ ? a.n_first - m : a.n_first + m;
      const bool last = m + 1 == a.count;
      if (!ADJ && to_snap-- == 0) {
        snapshot(m, n);
        to_snap = a.segment - 1;
      }
      // opaque copies: what is derived from them row by row is computed where it is used, not kept in
      // registers over the steps
      int dpo = dp, dl = dld, first_cell = cell0;
      asm volatile("" : "+r"(dpo), "+r"(dl), "+r"(first_cell));
      if (need_up) wait_halo(0, m);
      if (need_dn) wait_halo(1, m);
      const T* pc = buf + (m % NL) * BS + po0;
      const int level = (m + 1) % NL;
      T* pn = buf + level * BS + po0;
      const int older = NL == 2 ? 0 : ((m + 2) % NL - level) * BS;  // from the new level to the one before the current
      const T *ca_p = co_a, *cb_p = co_b;
      T wv[2 * R + 1][VZ];
#pragma unroll
      for (int q = 0; q < 2 * R; ++q) vload<T, VZ>(pc + (q - R) * dpo, wv[q]);
      const unsigned now = (ADJ ? inject && phase_c == 0 : a.src_corner != nullptr) ? rare : 0u;
      [[maybe_unused]] T* lps = lpo;
      [[maybe_unused]] int off = PF * dl;  // from the march's first row to the next one whose Lap p is loaded
      const bool first = n == 0 && (ADJ || a.first_b_one);
      // what a row reads of the levels: with registers to spare, the next row's while this one is computed
      // (its stores would hold the compiler's own loads back)
      constexpr bool AHEAD = RX <= (ADJ ? 2 : 4);
      T in_w[VZ], in_p[VZ], in_a[VZ], in_b[VZ];
      Row3<T, VZ> in_s;
      auto read_row = [&]() {
        vload<T, VZ>(pc + R * dpo, in_w);
        load_sides<T, R, VZ>(pc, in_s);
        vload<T, VZ>(pn + older, in_p);
        if constexpr (LAYER) {
          vload<T, VZ>(ca_p, in_a);
          vload<T, VZ>(cb_p, in_b);
          ca_p += co_d;
          cb_p += co_d;
        }
        pc += dpo;
        pn += dpo;
      };
      if (AHEAD && work) read_row();
#pragma unroll
      for (int k = 0; k < RX; ++k) {
        if (k >= nr) break;
        if (!AHEAD) read_row();
        Row3<T, VZ> rw = in_s;
        T pv[VZ], o[VZ], lp[VZ], two[VZ], ca[VZ], cb[VZ];
        T* out = pn - dpo;
#pragma unroll
        for (int v = 0; v < VZ; ++v) {
          wv[2 * R][v] = in_w[v];
          pv[v] = in_p[v];
          if (LAYER) { ca[v] = in_a[v]; cb[v] = in_b[v]; }
        }
        if (AHEAD && k + 1 < RX && k + 1 < nr) read_row();
        if constexpr (LAYER) {
          if (first) {  // B = 1 on Cerjan's first step; A does not apply to the adjoint's level 0
#pragma unroll
            for (int v = 0; v < VZ; ++v) (ADJ ? ca : cb)[v] = T(1);
          }
#pragma unroll
          for (int v = 0; v < VZ; ++v) cb[v] = -cb[v];
        }
#pragma unroll
        for (int v = 0; v < VZ; ++v) rw.c[v] = wv[R][v];
        lap_row<T, R, VZ>(wv, rw, a, lp);
        v_add(wv[R], wv[R], two);
        if constexpr (LAYER) v_fma(cb, pv, two, two);
        else v_fma(a.minus_one, pv, two, two);
        if constexpr (ADJ) {
          if (now >> k & 1u) {  // cotangents at touched cells
            const unsigned mp = map[(r0 + dir * k) * a.nv + vec];
            const T* cv = c_val + (m & 1) * a.cap_list + (mp >> 4);
#pragma unroll
            for (int v = 0; v < VZ; ++v)
              if (mp >> v & 1u) lp[v] = add_rn(lp[v], *cv++);
          }
        }
        v_fma(cc[C_REG ? k : k % PF], lp, two, o);
        if constexpr (!ADJ && LAYER) {
          if (now >> k & 1u) add_source(r0 + dir * k, m, o);
        }
        if constexpr (LAYER) v_mul(ca, o, o);
        vstore<T, VZ>(out, o);
        if constexpr (!ADJ) {
          if (lps) {  // (whole vectors: nothing reads the ghost columns of a stored Laplacian)
            vstore<T, VZ>(lps, lp);
            lps += dl;
          }
        } else {
          if (lap_now) {
            v_fma(wv[R], lpb[k % PF], gs[k], gs[k]);
            if (k + PF < RX && k + PF < nr) vldcg<T, VZ>(lap_now + off, lpb[k % PF]);
          }
          if (!C_REG && k + PF < RX && k + PF < nr) vldg<T, VZ>(a.C + first_cell + off, cc[k % PF]);
          off += dl;
        }
        if (k == R - 1 && !last && early) {  // the slab's edge rows are done: on their way while the rest is stepped
          if (send_up) send_rows(0, false, m, level);
          if (send_dn) send_rows(1, true, m, level);
        }
#pragma unroll
        for (int q = 0; q < 2 * R; ++q)
#pragma unroll
          for (int v = 0; v < VZ; ++v) wv[q][v] = wv[q + 1][v];
      }
      if (!early) {
        if constexpr (IMP) impose(m, level);
        else if (!ADJ && !LAYER && now) {  // the source, onto the stored cells (A = 1)
          for (unsigned left = now; left; left &= left - 1) {
            const int r = r0 + dir * (__ffs(left) - 1);
            T* row = buf + level * BS + (R + r) * pitch + zc;
            T o[VZ];
            vload<T, VZ>(row, o);
            add_source(r, m, o);
            vstore<T, VZ>(row, o);
          }
        }
        if (send_up && !last) send_rows(0, false, m, level);
        if (send_dn && !last) send_rows(1, true, m, level);
      }
      if (send_late && !last) send_rows(1, false, m, level);
      if constexpr (ADJ) {
        if (!last) {
          lap_now = lap_of(n - 1);
#pragma unroll
          for (int k = 0; k < PF && k < RX; ++k) {
            if (lap_now && k < nr) vldcg<T, VZ>(lap_now + k * dl, lpb[k]);
            if (!C_REG && k < nr) vldg<T, VZ>(a.C + first_cell + k * dl, cc[k]);
          }
        }
        if (--phase_c < 0) phase_c = a.substeps - 1;
      } else if (lpo) {
        lpo += a.level;
      }
      cta_barrier();
    }
  };

  // The steps of a strip with layer cells of a PML (pml2d.cuh has the formulas). The strip marches down with the
  // x faces above the row (old and new values) carried from the row before; a row computes its own z faces and
  // the next vector's first, whose old value it reads from the other step parity's array.
  auto pml_steps = [&]() {
    if constexpr (PML) {
      const int w = ne + 3, fs = (a.max_rows + 1) * w * VZ;
      const int slot = edge_vec ? (vec < a.edge_lo ? vec : vec - a.edge_hi + a.edge_lo + 1) : w - 1;
      const int fifth = edge_vec ? VZ : 0;
      T* lpo = !ADJ && a.lap_out ? a.lap_out + so + cell0 : nullptr;
      int phase_c = phase, to_snap = snap0;
      for (int m = 0; m < a.count; ++m) {
        const int n = ADJ ? a.n_first - m : a.n_first + m;
        const bool last = m + 1 == a.count;
        if (!ADJ && to_snap-- == 0) {
          if (work) snapshot(m, n);
          to_snap = a.segment - 1;
        }
        int dpo = pitch, dl = ld, first_cell = cell0;
        asm volatile("" : "+r"(dpo), "+r"(dl), "+r"(first_cell));
        if (need_up) wait_halo(0, m);
        if (need_dn) wait_halo(1, m);
          const int level = (m + 1) % NL;
        const T* pc = buf + (m % NL) * BS + po0;
        T* pn = buf + level * BS + po0;
        const int older = NL == 2 ? 0 : ((m + 2) % NL - level) * BS;
        const T* co = pml_row + (r0 * w + slot) * VZ;
        T* f0 = psi0 + r0 * pitch + zc;
        const T* f1o = psi1 + ((m & 1) * a.max_rows + r0) * pitch + zc;
        T* f1n = psi1 + ((1 - (m & 1)) * a.max_rows + r0) * pitch + zc;
        const unsigned now = (ADJ ? inject && phase_c == 0 : a.src_corner != nullptr) ? rare : 0u;
        [[maybe_unused]] T* lps = lpo;
        [[maybe_unused]] int off = PF * dl;
        int cell = first_cell;
        T wv[2 * R + 1][VZ], pv[VZ], pvn[VZ], fo[VZ], fn[VZ];
#pragma unroll
        for (int q = 0; q < 2 * R; ++q) vload<T, VZ>(pc + (q - R) * dpo, wv[q]);
        // the coefficients of face row r (0: this row's, 1: the next row's)
        auto face_co = [&](int next, T (&al)[VZ], T (&be)[VZ]) {
          if (alike) {
            vload<T, VZ>(co + 3 * fs + next * w * VZ, al);
            vload<T, VZ>(co + 4 * fs + next * w * VZ, be);
          } else {
            vldg<T, VZ>(a.alpha[0] + cell + next * dl, al);
            vldg<T, VZ>(a.beta[0] + cell + next * dl, be);
          }
        };
        if (work) {  // the x faces above the first row
          T al[VZ], be[VZ];
          face_co(0, al, be);
          vload<T, VZ>(f0, fo);
          if constexpr (!ADJ) {
#pragma unroll
            for (int v = 0; v < VZ; ++v)
              fn[v] = fma_rn(be[v], add_rn(wv[R][v], -wv[R - 1][v]), mul_rn(al[v], fo[v]));
          } else {
            vload<T, VZ>(pn + older, pv);
            T pu[VZ];
            vload<T, VZ>(pn + older - dpo, pu);
#pragma unroll
            for (int v = 0; v < VZ; ++v)
              fn[v] = fma_rn(-a.hx2, add_rn(add_rn(wv[R][v], pv[v]), -add_rn(wv[R - 1][v], pu[v])), mul_rn(al[v], fo[v]));
          }
          vstore<T, VZ>(f0, fn);
          if constexpr (ADJ) {  // the adjoint needs beta times the new face
#pragma unroll
            for (int v = 0; v < VZ; ++v) fn[v] = mul_rn(be[v], fn[v]);
          }
        }
#pragma unroll
        for (int k = 0; k < RX; ++k) {
          if (k >= nr) break;
          // every read of the row before its stores (which would hold later reads back)
          const bool inner = k + 1 < nr;
          Row3<T, VZ> rw;
          T o[VZ], lp[VZ], px[VZ], jo[VZ], jn[VZ], al0[VZ], be0[VZ], al[VZ + 1], be[VZ + 1], zo[VZ + 1], zn[VZ + 1];
          T cA[VZ], cB[VZ], cZ[VZ], t[VZ], sl = T(0), sr = T(0);
          vload<T, VZ>(pc + R * dpo, wv[2 * R]);
          load_sides<T, R, VZ>(pc, rw);
          f0 += dpo;
          if (inner) vload<T, VZ>(f0, jo);
          else {
#pragma unroll
            for (int v = 0; v < VZ; ++v) jo[v] = f_end[v];
          }
          vload<T, VZ>(f1o, t);
#pragma unroll
          for (int v = 0; v < VZ; ++v) zo[v] = t[v];
          zo[VZ] = f1o[VZ];
          face_co(1, al0, be0);
          if (alike) {
            vload<T, VZ>(co + 5 * fs, t);
#pragma unroll
            for (int v = 0; v < VZ; ++v) al[v] = t[v];
            vload<T, VZ>(co + 6 * fs, t);
#pragma unroll
            for (int v = 0; v < VZ; ++v) be[v] = t[v];
            al[VZ] = co[5 * fs + fifth];
            be[VZ] = co[6 * fs + fifth];
            vload<T, VZ>(co, cA);
            vload<T, VZ>(co + fs, cB);
            vload<T, VZ>(co + 2 * fs, cZ);
          } else {
#pragma unroll
            for (int v = 0; v <= VZ; ++v) {
              al[v] = a.alpha[1][cell + v];
              be[v] = a.beta[1][cell + v];
            }
            vldg<T, VZ>(a.A + cell, cA);
            vldg<T, VZ>(a.B + cell, cB);
            vldg<T, VZ>(a.zz + cell, cZ);
          }
          if constexpr (!ADJ) {
            vload<T, VZ>(pn, pv);
          } else {
            vload<T, VZ>(pn + older + dpo, pvn);
            sl = pn[older - 1];
            sr = pn[older + VZ];
          }
#pragma unroll
          for (int v = 0; v < VZ; ++v) rw.c[v] = wv[R][v];
          lap_row<T, R, VZ>(wv, rw, a, lp);
          // x faces below the row
          if constexpr (!ADJ) {
#pragma unroll
            for (int v = 0; v < VZ; ++v) {
              jn[v] = fma_rn(be0[v], add_rn(wv[R + 1][v], -wv[R][v]), mul_rn(al0[v], jo[v]));
              px[v] = mul_rn(a.hx2, add_rn(add_rn(jn[v], jo[v]), -add_rn(fn[v], fo[v])));
            }
          } else {
#pragma unroll
            for (int v = 0; v < VZ; ++v)
              jn[v] = fma_rn(-a.hx2, add_rn(add_rn(wv[R + 1][v], pvn[v]), -add_rn(wv[R][v], pv[v])), mul_rn(al0[v], jo[v]));
          }
          // z faces of the row's vector and the next one's first
          if constexpr (!ADJ) {
#pragma unroll
            for (int v = 0; v <= VZ; ++v)
              zn[v] = fma_rn(be[v], add_rn(zval(rw, v), -zval(rw, v - 1)), mul_rn(al[v], zo[v]));
#pragma unroll
            for (int v = 0; v < VZ; ++v)
              px[v] = fma_rn(a.hz2, add_rn(add_rn(zn[v + 1], zo[v + 1]), -add_rn(zn[v], zo[v])), px[v]);
          } else {
            T sz[VZ + 2];  // q^{k+1} + q^{k+2} at columns -1 .. VZ
            sz[0] = add_rn(zval(rw, -1), sl);
            sz[VZ + 1] = add_rn(zval(rw, VZ), sr);
#pragma unroll
            for (int v = 0; v < VZ; ++v) sz[v + 1] = add_rn(wv[R][v], pv[v]);
#pragma unroll
            for (int v = 0; v <= VZ; ++v)
              zn[v] = fma_rn(-a.hz2, add_rn(sz[v + 1], -sz[v]), mul_rn(al[v], zo[v]));
          }
          if (inner) vstore<T, VZ>(f0, jn);
          else {
#pragma unroll
            for (int v = 0; v < VZ; ++v) f_end[v] = jn[v];
          }
#pragma unroll
          for (int v = 0; v < VZ; ++v) t[v] = zn[v];
          vstore<T, VZ>(f1n, t);
          if (vec == a.nv - 1) f1n[VZ] = zn[VZ];  // face P1, where it starts a vector
#pragma unroll
          for (int v = 0; v < VZ; ++v) {
            if constexpr (ADJ) {
              jn[v] = mul_rn(be0[v], jn[v]);
              px[v] = add_rn(add_rn(jn[v], -fn[v]), add_rn(mul_rn(be[v + 1], zn[v + 1]), -mul_rn(be[v], zn[v])));
            }
            fo[v] = jo[v];
            fn[v] = jn[v];
          }
          if constexpr (!ADJ) {
#pragma unroll
            for (int v = 0; v < VZ; ++v) {
              lp[v] = add_rn(lp[v], px[v]);
              o[v] = fma_rn(-cZ[v], wv[R][v], fma_rn(cc[k][v], lp[v], fma_rn(-cB[v], pv[v], add_rn(wv[R][v], wv[R][v]))));
            }
            if (now >> k & 1u) add_source(r0 + k, m, o);
#pragma unroll
            for (int v = 0; v < VZ; ++v) o[v] = mul_rn(cA[v], o[v]);
            if (lps) {
              vstore<T, VZ>(lps, lp);
              lps += dl;
            }
          } else {
            if (now >> k & 1u) {  // cotangents at touched cells
              const unsigned mp = map[(r0 + k) * a.nv + vec];
              const T* cv = c_val + (m & 1) * a.cap_list + (mp >> 4);
#pragma unroll
              for (int v = 0; v < VZ; ++v)
                if (mp >> v & 1u) lp[v] = add_rn(lp[v], *cv++);
            }
#pragma unroll
            for (int v = 0; v < VZ; ++v) {
              o[v] = fma_rn(cc[k][v], add_rn(lp[v], -px[v]),
                            fma_rn(-cB[v], pv[v], fma_rn(-cZ[v], wv[R][v], add_rn(wv[R][v], wv[R][v]))));
              if (n >= 1) o[v] = mul_rn(cA[v], o[v]);
              pv[v] = pvn[v];
            }
            if (lap_now) {
              v_fma(wv[R], lpb[k % PF], gs[k], gs[k]);
              if (k + PF < RX && k + PF < nr) vldcg<T, VZ>(lap_now + off, lpb[k % PF]);
            }
            off += dl;
          }
          vstore<T, VZ>(pn, o);
          if (k == R - 1 && !last && early && send_up) send_rows(0, false, m, level);
          pc += dpo;
          pn += dpo;
          f1o += dpo;
          f1n += dpo;
          co += w * VZ;
          cell += dl;
#pragma unroll
          for (int q = 0; q < 2 * R; ++q)
#pragma unroll
            for (int v = 0; v < VZ; ++v) wv[q][v] = wv[q + 1][v];
        }
        if (!early) {
          if constexpr (IMP) impose(m, level);
          if (send_up && !last) send_rows(0, false, m, level);
        }
        if (send_late && !last) send_rows(1, false, m, level);
        if constexpr (ADJ) {
          if (!last) {
            lap_now = lap_of(n - 1);
#pragma unroll
            for (int k = 0; k < PF && k < RX; ++k)
              if (lap_now && k < nr) vldcg<T, VZ>(lap_now + k * dl, lpb[k]);
          }
          if (--phase_c < 0) phase_c = a.substeps - 1;
        } else if (lpo) {
          lpo += a.level;
        }
        cta_barrier();
      }
    }
  };

  if (tid >= svc) {  // the service warps
    const int id = tid - svc, ns = nthr - svc;
    T wave = T(0), weight = T(0);  // threads 0..3: the next step's wavelet value, loaded a step ahead
    const bool src = !ADJ && a.src_corner && id < 4;
    if (src) {
      weight = a.src_w[4 * s + id];
      if (a.count > 1) wave = a.wavelet[a.n_first + 1];
    }
    for (int m = 0; m < a.count; ++m) {
      const int n = ADJ ? a.n_first - m : a.n_first + m;
      const bool last = m + 1 == a.count, rec = phase == 0;
      // the next step's halos are expected (after a wait that gave up, the phase before may not have completed)
      if (id == 0 && !last && !*(volatile int*)&gave_up) {
        const unsigned tx = R * a.nv * 16, b = mbar_a + 8 * ((m + 1) & 1);
        if (has_up) mbar_expect(b, tx + (sampled ? 16 : 0));
        if (has_dn) mbar_expect(b + 16, tx);
      }
      if constexpr (ADJ) {
        const int np = n - 2;  // Lap p of the step after the next, this slab's rows in one piece, to L2
        if (id == 0 && np >= a.lap_n0 && np < a.lap_end && m + 2 < a.count) {
          const T* src = a.lap + (long long)(np - a.lap_n0) * a.level + so + g.origin + (long long)X0 * ld;
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(rows * ld * (int)sizeof(T)) : "memory");
        }
        if (--phase < 0) { phase = a.substeps - 1; --j; }
        if (inject && phase == 0 && !last) cotangents(j, c_val + (1 - (m & 1)) * a.cap_list, id, ns);
      } else {
        const T* P = buf + (m % NL) * BS;
        auto sample = [&](int e) {  // a receiver of p^n
          const T* p0 = P + l_off[e];
          const T* w = l_w + 4 * e;
          T v = mul_rn(w[0], p0[0]);
          v = fma_rn(w[1], p0[1], v);
          v = fma_rn(w[2], p0[pitch], v);
          v = fma_rn(w[3], p0[pitch + 1], v);
          a.traces[(long long)s * a.n_rec * a.n_t + l_id[e] + j] = v;
        };
        if (sampled && id < 32) {
          const int n_edge = rec ? count[1] : 0;
          // The wait is not for the samples alone: the piece below counts towards the phase of step m + 1, which
          // shares its mbarrier with that of m - 1, and only the rows this waits for say that the CTA below has
          // seen m - 1 complete.
          if (has_dn && (n_edge > 0 || !last)) wait_halo(1, m);
          for (int e = id; e < n_edge; e += 32) sample(a.cap_list - 1 - e);
          __syncwarp();
          if (id == 0 && has_dn && !last && !dead)
            send_bytes(smem_addr(buf) + dn_off + a.nv * 16 + ((m + 1) % NL) * (unsigned)(BS * (int)sizeof(T)),
                       smem_addr(buf) - 16, 16, mbar_a + dn_off + 8 * ((m + 1) & 1));
        }
        if (rec && sampled)
          for (int e = id, n_in = count[0]; e < n_in; e += ns) sample(e);
        if (src && !last) {  // the next step's source values, by step parity
          src_sh[4 * (1 - (m & 1)) + id] = mul_rn(weight, wave);
          if (m + 2 < a.count) wave = a.wavelet[n + 2];
        }
        if constexpr (IMP) if (!last) imposed_values(n + 2, i_val + (1 - (m & 1)) * a.n_imposed, id, ns);
        if (++phase == a.substeps) { phase = 0; ++j; }
      }
      cta_barrier();
    }
  } else if (layer_warp) {
    if constexpr (PML) pml_steps();
    else steps(std::true_type{});
  } else {
    steps(std::false_type{});
  }

  if (*(volatile int*)&gave_up && tid < a.cluster)
    asm volatile("st.shared::cluster.u32 [%0], %1;\n" ::"r"(map_cta(smem_addr(&lost_sh), tid)), "r"(1) : "memory");
  cluster_barrier();
  const bool lost = *(volatile int*)&lost_sh != 0;

  // ---- the last two levels (and the gradient sums) back to memory
  if (work && (a.out_cur || ADJ)) {
    const T* P = buf + (a.count % NL) * BS;             // the newest level
    const T* Q = buf + ((a.count + NL - 1) % NL) * BS;  // the one before
#pragma unroll
    for (int k = 0; k < RX; ++k)
      if (k < nr) {
        const long long o = so + cell0 + k * dld;
        T v0[VZ];
        vload<T, VZ>(P + po0 + k * dp, v0);
        store_row<T, VZ>(a.out_cur + o, v0, zc, g.n1);
        vload<T, VZ>(Q + po0 + k * dp, v0);
        store_row<T, VZ>(a.out_prev + o, v0, zc, g.n1);
        if constexpr (ADJ) {
          if (a.acc) store_row<T, VZ>(a.acc + o, gs[k], zc, g.n1);
        }
        if constexpr (PML) {  // the face fields (P1 + 1 faces in a row; face P0 from the last strip)
          const int r = r0 + dir * k;
          vload<T, VZ>(psi0 + r * pitch + zc, v0);
          store_row<T, VZ>(a.f_out[0] + o, v0, zc, g.n1);
          const T* f1 = psi1 + ((a.count & 1) * a.max_rows + r) * pitch + zc;
          vload<T, VZ>(f1, v0);
          store_row<T, VZ>(a.f_out[1] + o, v0, zc, g.n1 + 1);
          if (zc + VZ == g.n1) a.f_out[1][o + VZ] = f1[VZ];
        }
      }
    if constexpr (PML) {
      if (X0 + rb == g.n0) store_row<T, VZ>(a.f_out[0] + so + cell0 + (long long)nr * ld, f_end, zc, g.n1);
    }
  }
  if (lost) mark_lost<T, VZ, ADJ>(a, s, (long long)s * g.field + cell0, nr, dld, zc, g.n1);
  cluster_barrier();  // no CTA leaves while a neighbour may still address its shared memory
}

}  // namespace nw
