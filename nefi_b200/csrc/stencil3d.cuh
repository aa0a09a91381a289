// stencil3d.cuh — plane-marching 3-D leapfrog step for sm_100a (forward and q-form adjoint).
//
// A CTA of 256 threads owns a (y, z) tile of `ty` rows by `wv` 16-byte vectors of columns (chosen by the
// host so that the tiles divide the row evenly: 7 x 36 vectors on 288 columns) and marches along x over a
// chunk of planes. Thread t owns vector t % wv of row t / wv. Every plane the march touches passes once
// through a ring of R + 3 shared-memory tiles, (ty + 2R) rows by wv + 2 vectors (the y/z halo), staged by
// cp.async two planes ahead of its first use (one barrier per plane: a plane's copy is issued right after
// the barrier that frees its slot); the x-neighbours of a thread's cells stay in a (2R+1)-plane register
// window, fed from the ring when a plane arrives. The y/z neighbours of the centre plane come from its
// shared tile. Planes outside the grid are never copied: their window values are zero, like the ghost planes
// they stand for. C, p^{n-1} (q^{n+2}), the stored Lap p and the gradient accumulator are read at the
// thread's own cells straight from global memory with vector loads issued one plane ahead; A/B (layer
// cells) when needed.
//
// The step is bound by issue and latency before DRAM: 8-byte vectors on fixed 8 x 64 tiles took 237 us for
// a forward step of two 288^3 instances (10 % of the lanes past the row), 16-byte ones on fitted tiles
// 181 us (of two 288^3 instances; 4.0 TB/s of the 16 bytes a cell-update needs, C shared by the instances).
#pragma once
#include "kernels.cuh"
#include "stencil2d.cuh"
#include "lanes.cuh"

namespace nw {

template <typename T, int R>
struct Tile3Shape {
  static constexpr int NT = 256;
  static constexpr int VZ = 16 / (int)sizeof(T);   // columns of a vector
  static constexpr int NCH = 2;                    // copied chunks per thread and plane: (ty + 2R) (wv + 2) <= 512
  static constexpr int NSP = R + 3;                // planes in the ring
  __host__ __device__ static int row(int wv) { return (wv + 2) * VZ; }
  __host__ __device__ static int plane(int wv, int ty) { return (ty + 2 * R) * row(wv); }
};

template <typename T, int R, bool ADJ>
__global__ void __launch_bounds__(Tile3Shape<T, R>::NT, 3) step3t(const __grid_constant__ KGrid<T> g, const __grid_constant__ Step3<T> a, int wv_, int ty, int xc, int n_shots) {
  using S = Tile3Shape<T, R>;
  constexpr int NSP = S::NSP, VZ = S::VZ;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);  // [NSP][PS]
  const int SW = S::row(wv_), PS = S::plane(wv_, ty);

  // grid.x = tile * n_shots + shot (the shot fastest, so that the CTAs of one tile for all shots run
  // together and the shot-independent fields C, A, B come from L2 after the first), grid.y = x chunk
  const int n_vec = (g.n2 + VZ - 1) / VZ, tiles_z = (n_vec + wv_ - 1) / wv_;
  const int s = blockIdx.x % n_shots, tile = blockIdx.x / n_shots;
  const int z0 = (tile % tiles_z) * wv_ * VZ, y0 = (tile / tiles_z) * ty;
  const int x0 = blockIdx.y * xc, x1 = min(x0 + xc, g.n0);
  const long long so = (long long)s * g.field;
  const int trow = threadIdx.x / wv_, vec = threadIdx.x - trow * wv_;
  const int y = y0 + trow, zc = z0 + vec * VZ;
  const bool own = trow < ty && y < g.n1 && zc < g.n2;
  const int ld = (int)g.s1;
  const T* __restrict__ cur = a.cur + so;
  // The chunks of one plane tile: element offsets from the field base for plane 0 (add x * s0 for plane x;
  // they are >= 0 for x >= 0 thanks to the ghost planes and the guard, and -1 marks a chunk that is not
  // copied); rows and columns that no output cell reads (beyond the ghost rows, past the row pitch) are not
  // copied.
  CopyPlan<S::NCH> pp;
#pragma unroll
  for (int i = 0; i < S::NCH; ++i) {
    const int c = threadIdx.x + S::NT * i;
    const int row = c / (wv_ + 2), ch = c - row * (wv_ + 2);
    const int yy = y0 - R + row, zz = z0 + (ch - 1) * VZ;
    pp.soff[i] = (unsigned)((row * SW + ch * VZ) * (int)sizeof(T));
    pp.goff[i] = (row < ty + 2 * R && yy < g.n1 + R && zz < ld) ? (int)(g.origin + (long long)yy * ld + zz) : -1;
  }
  // the planes of the march: xa = x0 - R .. xb - 1 = x1 + R - 1; plane p sits in ring slot
  // (p - xa) % NSP. When plane p is consumed (its own cells enter the window front) the centre is
  // p - R: planes p - R .. p must be resident, and the copy of plane p + 2 goes into the slot of
  // plane p - R - 1 (NSP = R + 3), the centre of the previous iteration.
  const int xa = x0 - R, xb = x1 + R;
  const unsigned ring_sa = smem_addr(ring), plane_b = (unsigned)(PS * (int)sizeof(T));
  auto issue_plane = [&](int p, int slot) {
    if (p >= 0 && p < g.n0 && p < xb) issue(pp, cur + (long long)p * g.s0, ring_sa + slot * plane_b);
  };
  wait_previous_grid();
  allow_next_grid();
  if (!ADJ && a.traces)
    gather_receivers<T, 8>(cur, a.traces, a.rec_idx, a.rec_w, a.n_rec, a.n_t, a.j, s,
                           ((long long)blockIdx.y * (gridDim.x / n_shots) + tile) * blockDim.x + threadIdx.x,
                           (long long)(gridDim.x / n_shots) * gridDim.y * blockDim.x);
  issue_plane(xa, 0);  // one commit group per plane, empty groups included
  cp_async_commit();
  issue_plane(xa + 1, 1);
  cp_async_commit();
  const bool yz_layer = y0 < g.lo1 || y0 + ty > g.hi1 || z0 < g.lo2 || z0 + wv_ * VZ > g.hi2;
  // source corners of this shot (forward)
  int bx = -4, by = -4, bz = -4;
  if (!ADJ && a.src_corner) { bx = a.src_corner[3 * s]; by = a.src_corner[3 * s + 1]; bz = a.src_corner[3 * s + 2]; }

  T wv[2 * R + 1][VZ];  // own cells of planes p - 2R .. p
#pragma unroll
  for (int q = 0; q < 2 * R + 1; ++q)
#pragma unroll
    for (int v = 0; v < VZ; ++v) wv[q][v] = T(0);
  const int own_off = (trow + R) * SW + (vec + 1) * VZ;
  // the per-cell fields of the next plane's own cells, loaded one plane ahead into registers
  long long i_next = g.origin + (long long)x0 * g.s0 + (long long)y * ld + zc;  // of the next plane prefetched
  T pvn[VZ], ccn[VZ], gln[VZ], ggn[VZ];
  auto prefetch = [&](int x) {
    if (x < x1 && own) {
      vldg<T, VZ>(a.prev + so + i_next, pvn);
      vldg<T, VZ>(a.C + i_next, ccn);
      if (ADJ && a.lap) {
        vldg<T, VZ>(a.lap + so + i_next, gln);
        vload<T, VZ>(a.grad + so + i_next, ggn);
      }
    }
    i_next += g.s0;
  };
  prefetch(x0);
  int slot = 0;  // of plane p
  for (int p = xa; p < xb; ++p) {
    cp_async_wait<1>();  // this thread's copies of plane p have landed
    __syncthreads();     // everyone's have, and every thread is done with the previous centre's slot
    issue_plane(p + 2, slot + 2 >= NSP ? slot + 2 - NSP : slot + 2);  // into that slot
    cp_async_commit();
    if (p >= 0 && p < g.n0 && own) vload<T, VZ>(ring + slot * PS + own_off, wv[2 * R]);
    else {
#pragma unroll
      for (int v = 0; v < VZ; ++v) wv[2 * R][v] = T(0);
    }
    const int x = p - R;
    if (x >= x0 && own) {
      const T* P = ring + (slot >= R ? slot - R : slot - R + NSP) * PS + own_off;  // the centre plane's tile
      const long long i = i_next - g.s0;
      Row3<T, VZ> rw;
      load_sides<T, R, VZ>(P, rw);
#pragma unroll
      for (int v = 0; v < VZ; ++v) rw.c[v] = wv[R][v];
      T ym[VZ], yp[VZ], ym2[VZ], yp2[VZ];
      vload<T, VZ>(P - SW, ym);
      vload<T, VZ>(P + SW, yp);
      if (R == 2) {
        vload<T, VZ>(P - 2 * SW, ym2);
        vload<T, VZ>(P + 2 * SW, yp2);
      }
      T pv[VZ], cc[VZ], gl[VZ], gg[VZ];
#pragma unroll
      for (int v = 0; v < VZ; ++v) {
        pv[v] = pvn[v];
        cc[v] = ccn[v];
        gl[v] = gln[v];
        gg[v] = ggn[v];
      }
      prefetch(x + 1);  // in flight while this plane is computed
      T lap[VZ], t[VZ], o[VZ];
      v_mul(lane_weight(g.wc), wv[R], lap);
      v_add(wv[R - 1], wv[R + 1], t);
      v_fma(lane_weight(g.w1a), t, lap, lap);
      v_add(ym, yp, t);
      v_fma(lane_weight(g.w1b), t, lap, lap);
#pragma unroll
      for (int v = 0; v < VZ; ++v) t[v] = add_rn(zval(rw, v - 1), zval(rw, v + 1));
      v_fma(lane_weight(g.w1c), t, lap, lap);
      if constexpr (R == 2) {
        v_add(wv[0], wv[4], t);
        v_fma(lane_weight(g.w2a), t, lap, lap);
        v_add(ym2, yp2, t);
        v_fma(lane_weight(g.w2b), t, lap, lap);
#pragma unroll
        for (int v = 0; v < VZ; ++v) t[v] = add_rn(zval(rw, v - 2), zval(rw, v + 2));
        v_fma(lane_weight(g.w2c), t, lap, lap);
      }
      v_add(wv[R], wv[R], o);
      const bool layer = a.A && (yz_layer || x < g.lo0 || x >= g.hi0);
      if (layer && (ADJ || !a.b_one)) {
        T cb[VZ];
        vldg<T, VZ>(a.B + i, cb);
#pragma unroll
        for (int v = 0; v < VZ; ++v) cb[v] = -cb[v];
        v_fma(cb, pv, o, o);
      } else {
        v_fma(lane_weight(T(-1)), pv, o, o);
      }
      v_fma(cc, lap, o, o);
      if (!ADJ && bx >= x - 1 && bx <= x && by >= y - 1 && by <= y) {  // the source stencil touches this row
        const T wn = a.wavelet[a.n];
#pragma unroll
        for (int v = 0; v < VZ; ++v) {
          const int dx = x - bx, dy = y - by, dz = zc + v - bz;
          if (dz >= 0 && dz <= 1) o[v] = add_rn(o[v], mul_rn(a.src_w[8 * s + 4 * dx + 2 * dy + dz], wn));
        }
      }
      if (layer && (!ADJ || a.apply_a)) {
        T ca[VZ];
        vldg<T, VZ>(a.A + i, ca);
        v_mul(ca, o, o);
      }
      store_row<T, VZ>(a.next + so + i, o, zc, g.n2);
      if (!ADJ && a.lap_out) store_row<T, VZ>(a.lap_out + so + i, lap, zc, g.n2);
      if (ADJ && a.lap) {
        v_fma(wv[R], gl, gg, gg);
        store_row<T, VZ>(a.grad + so + i, gg, zc, g.n2);
      }
    }
    if (++slot == NSP) slot = 0;
#pragma unroll
    for (int q = 0; q < 2 * R; ++q)
#pragma unroll
      for (int v = 0; v < VZ; ++v) wv[q][v] = wv[q + 1][v];
  }
}

}  // namespace nw
