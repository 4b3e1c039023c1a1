// Brick lists of the FP64 tensor-core contractions, built on the device from
// the sphere lists, and the orchestration of those contractions.
//
// Two tilings of the home cell are made per orbital set: bricks of 128 points
// for the density (points are the MMA's 128 rows) and of 64 for the matrix
// elements (points are its K).  A sphere point's unrolled brick (home brick +
// period) falls in a small box per atom; flags over those boxes give the
// images of every home brick without sorting the points: mark, count per
// brick, scan, fill, and one rank sort per brick by (atom, unrolled brick),
// which fixes the order of all later sums.
#include <cuda_runtime.h>

#include <cmath>

#include "lcp_api_state.h"

namespace lcp {

namespace {

struct BoxDev {
  int32_t lo[3], ext[3];
  int64_t off;  // first flag of the atom
};

struct BuildGeom {
  int32_t ng[3], bd[3], nb[3];
  int32_t natom, P;
  const int64_t* sph_off;
  const int32_t* glist;
  const int32_t* clist;
  const int32_t* ijk;
};

__device__ __forceinline__ int floor_div(int a, int b) {
  const int q = a / b;
  return q - (a % b < 0 ? 1 : 0);
}

// Unrolled brick coordinates of sphere entry k and its slot within the brick.
__device__ __forceinline__ int point_brick(const BuildGeom& g, int64_t k, int c[3]) {
  const int gi = g.glist[k], cell = g.clist[k];
  const int plane = g.ng[1] * g.ng[2];
  const int x0 = gi / plane, x1 = (gi - x0 * plane) / g.ng[2], x2 = gi - x0 * plane - x1 * g.ng[2];
  const int x[3] = {x0, x1, x2};
  int slot = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int h = x[d] / g.bd[d];
    c[d] = g.ijk[cell * 3 + d] * g.nb[d] + h;
    slot = slot * g.bd[d] + (x[d] - h * g.bd[d]);
  }
  return slot;
}

// Bounding box of each atom's unrolled bricks: box[atom][min 0..2, max 3..5].
__global__ void __launch_bounds__(256) f64_box_kernel(BuildGeom g, int32_t* __restrict__ box) {
  const int a = blockIdx.y;
  int mn[3] = {1 << 30, 1 << 30, 1 << 30}, mx[3] = {-(1 << 30), -(1 << 30), -(1 << 30)};
  for (int64_t k = g.sph_off[a] + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < g.sph_off[a + 1];
       k += (int64_t)gridDim.x * blockDim.x) {
    int c[3];
    point_brick(g, k, c);
    for (int d = 0; d < 3; ++d) {
      mn[d] = min(mn[d], c[d]);
      mx[d] = max(mx[d], c[d]);
    }
  }
  for (int d = 0; d < 3; ++d) {
    const int lo = __reduce_min_sync(0xffffffffu, mn[d]), hi = __reduce_max_sync(0xffffffffu, mx[d]);
    if ((threadIdx.x & 31) == 0 && lo <= hi) {
      atomicMin(box + a * 6 + d, lo);
      atomicMax(box + a * 6 + 3 + d, hi);
    }
  }
}

__device__ __forceinline__ int64_t box_index(const BoxDev& b, const int c[3]) {
  return b.off + ((int64_t)(c[0] - b.lo[0]) * b.ext[1] + (c[1] - b.lo[1])) * b.ext[2] + (c[2] - b.lo[2]);
}

__global__ void __launch_bounds__(256) f64_mark_kernel(BuildGeom g, const BoxDev* __restrict__ box,
                                                       int32_t* __restrict__ flag) {
  const int a = blockIdx.y;
  const BoxDev b = box[a];
  for (int64_t k = g.sph_off[a] + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < g.sph_off[a + 1];
       k += (int64_t)gridDim.x * blockDim.x) {
    int c[3];
    point_brick(g, k, c);
    flag[box_index(b, c)] = 1;
  }
}

// Unrolled brick of box entry e of an atom and its home brick.
__device__ __forceinline__ int64_t box_brick(const BuildGeom& g, const BoxDev& b, int64_t e, int c[3]) {
  c[2] = (int)(e % b.ext[2]) + b.lo[2];
  c[1] = (int)(e / b.ext[2] % b.ext[1]) + b.lo[1];
  c[0] = (int)(e / ((int64_t)b.ext[2] * b.ext[1])) + b.lo[0];
  int64_t hb = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) hb = hb * g.nb[d] + (c[d] - floor_div(c[d], g.nb[d]) * g.nb[d]);
  return hb;
}

// FILL = false: images per home brick; true: their keys (atom << 32 | box entry).
template <bool FILL>
__global__ void __launch_bounds__(256) f64_images_kernel(BuildGeom g, const BoxDev* __restrict__ box,
                                                         const int32_t* __restrict__ numorbs,
                                                         const int32_t* __restrict__ flag, int32_t* __restrict__ cnt,
                                                         const int64_t* __restrict__ img_off,
                                                         uint64_t* __restrict__ key) {
  const int a = blockIdx.y;
  const BoxDev b = box[a];
  if (numorbs[a] == 0) return;
  const int64_t n = (int64_t)b.ext[0] * b.ext[1] * b.ext[2];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    if (!flag[b.off + e]) continue;
    int c[3];
    const int64_t hb = box_brick(g, b, e, c);
    const int pos = atomicAdd(cnt + hb, 1);
    if (FILL) key[img_off[hb] + pos] = ((uint64_t)a << 32) | (uint64_t)e;
  }
}

// Per home brick (one warp): its images in key order, their first rows, and
// the sizes of its row and pair tables.
__global__ void __launch_bounds__(256) f64_sort_kernel(BuildGeom g, const BoxDev* __restrict__ box,
                                                       const int32_t* __restrict__ numorbs, int64_t nbricks,
                                                       const int64_t* __restrict__ img_off,
                                                       const uint64_t* __restrict__ key, int32_t* __restrict__ flag,
                                                       int32_t* __restrict__ img_atom, int4* __restrict__ img_per,
                                                       int32_t* __restrict__ img_row0, int32_t* __restrict__ row_cnt,
                                                       int32_t* __restrict__ chunk_cnt, int32_t* __restrict__ tab_cnt) {
  const int lane = threadIdx.x & 31;
  for (int64_t hb = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; hb < nbricks;
       hb += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int64_t i0 = img_off[hb];
    const int m = (int)(img_off[hb + 1] - i0);
    int rows = 0;
    for (int i = lane; i < m; i += 32) {
      const uint64_t my = key[i0 + i];
      int rank = 0, row0 = 0;
      for (int j = 0; j < m; ++j) {
        const uint64_t o = key[i0 + j];
        if (o < my) {
          ++rank;
          row0 += numorbs[o >> 32];
        }
      }
      const int a = (int)(my >> 32);
      const BoxDev b = box[a];
      const int64_t e = (int64_t)(my & 0xffffffffu);
      int c[3];
      box_brick(g, b, e, c);
      img_atom[i0 + rank] = a;
      img_per[i0 + rank] = make_int4(floor_div(c[0], g.nb[0]), floor_div(c[1], g.nb[1]), floor_div(c[2], g.nb[2]), 0);
      img_row0[i0 + rank] = row0;
      flag[b.off + e] = (int32_t)(i0 + rank) + 1;
      rows += numorbs[a];
    }
    rows = __reduce_add_sync(0xffffffffu, rows);
    if (lane == 0) {
      row_cnt[hb] = rows;
      chunk_cnt[hb] = (rows + 31) / 32;
      tab_cnt[hb] = m * m;
    }
  }
}

__global__ void __launch_bounds__(256) f64_slot_kernel(BuildGeom g, const BoxDev* __restrict__ box,
                                                       const int32_t* __restrict__ numorbs,
                                                       const int32_t* __restrict__ flag, int32_t* __restrict__ slot) {
  const int a = blockIdx.y;
  if (numorbs[a] == 0) return;
  const BoxDev b = box[a];
  const int64_t k0 = g.sph_off[a];
  for (int64_t k = k0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < g.sph_off[a + 1];
       k += (int64_t)gridDim.x * blockDim.x) {
    int c[3];
    const int s = point_brick(g, k, c);
    slot[((int64_t)flag[box_index(b, c)] - 1) * g.P + s] = (int32_t)(k - k0);
  }
}

// Pair tables: the ordered pair (atom_s, atom_t, R_s - R_t) of images s and t
// (matrix elements: s <= t only) by binary search in atom_s's list (the self pair first, then by neighbour
// and cell).
__global__ void __launch_bounds__(256) f64_tab_kernel(F64Pairs pr, int64_t nbricks,
                                                      const int64_t* __restrict__ img_off,
                                                      const int32_t* __restrict__ img_atom,
                                                      const int4* __restrict__ img_per,
                                                      const int64_t* __restrict__ tab_off, int elements,
                                                      int32_t* __restrict__ tab) {
  for (int64_t hb = blockIdx.x; hb < nbricks; hb += gridDim.x) {
    const int64_t i0 = img_off[hb];
    const int m = (int)(img_off[hb + 1] - i0);
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
      const int s = e / m, t = e - s * m;
      int32_t out = -1;
      if (s <= t || !elements) {
        const int as = img_atom[i0 + s], at = img_atom[i0 + t];
        const int4 rs = img_per[i0 + s], rt = img_per[i0 + t];
        const int d0 = rs.x - rt.x, d1 = rs.y - rt.y, d2 = rs.z - rt.z;
        const int C = pr.cpy, n = 2 * C + 1;
        int64_t p = -1;
        if (s == t) {
          p = pr.first[as];
        } else if (abs(d0) <= C && abs(d1) <= C && abs(d2) <= C) {
          const int64_t want = (int64_t)at * pr.ncell + pr.ratv[((d0 + C) * n + (d1 + C)) * n + (d2 + C)];
          int64_t lo = pr.first[as] + 1, hi = pr.first[as + 1];
          while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            const int64_t v = (int64_t)pr.jatom[mid] * pr.ncell + pr.cell[mid];
            if (v < want) lo = mid + 1;
            else hi = mid;
          }
          if (lo < pr.first[as + 1] && (int64_t)pr.jatom[lo] * pr.ncell + pr.cell[lo] == want) p = lo;
        }
        // images are sorted by (atom, period), so for s <= t the pair is the kept one of the two (or its own partner)
        if (p >= 0) out = (int32_t)pr.boff[elements ? pr.partner[p] : p];
      }
      tab[tab_off[hb] + e] = out;
    }
  }
}

__global__ void __launch_bounds__(256) f64_bricks_kernel(int64_t nbricks, const int64_t* __restrict__ img_off,
                                                         const int64_t* __restrict__ row_off,
                                                         const int64_t* __restrict__ chunk_off,
                                                         const int64_t* __restrict__ tab_off,
                                                         F64Brick* __restrict__ out) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nbricks; k += (int64_t)gridDim.x * blockDim.x) {
    F64Brick b;
    b.row = (uint32_t)row_off[k];
    b.chunk = (uint32_t)chunk_off[k];
    b.tab = (uint32_t)tab_off[k];
    b.size = (uint32_t)(row_off[k + 1] - row_off[k]) | ((uint32_t)(img_off[k + 1] - img_off[k]) << 16);
    out[k] = b;
  }
}

__global__ void f64_fill_kernel(int32_t* __restrict__ x, int64_t n, int32_t v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) x[i] = v;
}

// Brick sides of at most P points in all: the fewest products, taken as
// bricks x rows x (rows + 64) with a brick's rows from the Steiner formula
// (the volume of each cutoff sphere grown by the brick), so that ragged grids
// get sides that divide them.
// Returns the predicted rows per brick.
double choose_shape(const UCell& u, int P, int32_t* bd) {
  double len[3], vcell = u.gridvol * (double)u.nn(), best = 1e300, best_rows = 0.0;
  for (int d = 0; d < 3; ++d)
    len[d] = std::sqrt(u.glat[d][0] * u.glat[d][0] + u.glat[d][1] * u.glat[d][1] + u.glat[d][2] * u.glat[d][2]);
  for (int b0 = 1; b0 <= std::min(16, u.ngrid[0]); ++b0)
    for (int b1 = 1; b1 <= std::min(16, u.ngrid[1]) && b0 * b1 <= P; ++b1)
      for (int b2 = 1; b2 <= std::min(16, u.ngrid[2]) && b0 * b1 * b2 <= P; ++b2) {
        const int b[3] = {b0, b1, b2};
        double L[3], n = 1.0;
        for (int d = 0; d < 3; ++d) {
          L[d] = len[d] * (b[d] - 1);
          n *= (double)((u.ngrid[d] + b[d] - 1) / b[d]);
        }
        const double s2 = L[0] * L[1] + L[1] * L[2] + L[0] * L[2], s1 = L[0] + L[1] + L[2];
        double rows = 0.0;
        for (int a = 0; a < u.natom; ++a) {
          const double r = u.cut[a];
          rows += u.numorbs[a] * (L[0] * L[1] * L[2] + 2 * r * s2 + 3.14159265358979 * r * r * s1 +
                                  4.18879020478639 * r * r * r) / vcell;
        }
        const double cost = n * rows * (rows + 64.0);
        if (cost < best) {
          best = cost;
          best_rows = rows;
          for (int d = 0; d < 3; ++d) bd[d] = b[d];
        }
      }
  return best_rows;
}

int blocks_for(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 8)); }

// One tiling; *fits = false when a brick or a table is beyond the kernels' limits.
// Without the room for it, S.need is set and S holds nothing.
lcp_status build_set(lcp_ctx* ctx, lcp_orbs* o, const DBuf& ijk, F64Set& S, int P, bool* fits) {
  const UCell& u = o->ucell->u;
  cudaStream_t st = ctx->stream;
  F64Bricks& g = S.g;
  g = F64Bricks{};
  g.P = P;
  choose_shape(u, P, g.bdim);
  g.nbricks = 1;
  g.npts = 1;
  BuildGeom bg{};
  for (int d = 0; d < 3; ++d) {
    g.ngrid[d] = bg.ng[d] = u.ngrid[d];
    g.nb[d] = bg.nb[d] = (u.ngrid[d] + g.bdim[d] - 1) / g.bdim[d];
    bg.bd[d] = g.bdim[d];
    g.nbricks *= g.nb[d];
    g.npts *= g.bdim[d];
  }
  bg.natom = u.natom;
  bg.P = P;
  bg.sph_off = o->geom.sph_off;
  bg.glist = o->geom.glist;
  bg.clist = o->geom.clist;
  bg.ijk = ijk.as<int32_t>();
  const int32_t* no = o->geom.numorbs;
  int64_t most = 1;
  for (int a = 0; a < u.natom; ++a) most = std::max(most, u.sphere_off[a + 1] - u.sphere_off[a]);
  const dim3 pts((unsigned)std::min<int64_t>((most + 1023) / 1024, 256), (unsigned)u.natom);
  // boxes
  DBuf d_row_off, d_chunk_off, d_tab_off;
  DBuf d_box, d_boxes, d_flag, d_cnt, d_key, d_scan, d_per, d_row0, d_cc, d_tc;
  std::vector<int32_t> box(6 * (size_t)u.natom);
  for (size_t i = 0; i < box.size(); ++i) box[i] = i % 6 < 3 ? (1 << 30) : -(1 << 30);
  API_CUDA(upload(d_box, box, st), "upload");
  f64_box_kernel<<<pts, 256, 0, st>>>(bg, d_box.as<int32_t>());
  API_CUDA(cudaGetLastError(), "brick boxes");
  API_CUDA(cudaMemcpyAsync(box.data(), d_box.p, box.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, st), "D2H");
  API_CUDA(cudaStreamSynchronize(st), "brick boxes");
  std::vector<BoxDev> boxes(u.natom);
  int64_t nflag = 0, most_box = 1;
  for (int a = 0; a < u.natom; ++a) {
    int64_t vol = 1;
    for (int d = 0; d < 3; ++d) {
      boxes[a].lo[d] = box[a * 6 + d];
      boxes[a].ext[d] = std::max(0, box[a * 6 + 3 + d] - box[a * 6 + d] + 1);
      if (u.sphere_off[a + 1] == u.sphere_off[a]) boxes[a].ext[d] = 0;
      vol *= boxes[a].ext[d];
    }
    boxes[a].off = nflag;
    nflag += vol;
    most_box = std::max(most_box, vol);
  }
  const dim3 bxs((unsigned)std::min<int64_t>((most_box + 255) / 256, 256), (unsigned)u.natom);
  API_CUDA(upload(d_boxes, boxes, st), "upload");
  API_CUDA(d_flag.ensure(std::max<int64_t>(nflag, 1) * sizeof(int32_t)), "alloc");
  API_CUDA(cudaMemsetAsync(d_flag.p, 0, nflag * sizeof(int32_t), st), "memset");
  API_CUDA(d_cnt.ensure(g.nbricks * sizeof(int32_t)), "alloc");
  API_CUDA(cudaMemsetAsync(d_cnt.p, 0, g.nbricks * sizeof(int32_t), st), "memset");
  API_CUDA(S.img_off.ensure((g.nbricks + 1) * sizeof(int64_t)), "alloc");
  API_CUDA(d_row_off.ensure((g.nbricks + 1) * sizeof(int64_t)), "alloc");
  API_CUDA(d_chunk_off.ensure((g.nbricks + 1) * sizeof(int64_t)), "alloc");
  API_CUDA(d_tab_off.ensure((g.nbricks + 1) * sizeof(int64_t)), "alloc");
  API_CUDA(d_scan.ensure((scan_blocks(g.nbricks) + 1) * sizeof(int64_t)), "alloc");
  const BoxDev* dbx = d_boxes.as<BoxDev>();
  f64_mark_kernel<<<pts, 256, 0, st>>>(bg, dbx, d_flag.as<int32_t>());
  API_CUDA(cudaGetLastError(), "brick marks");
  f64_images_kernel<false><<<bxs, 256, 0, st>>>(bg, dbx, no, d_flag.as<int32_t>(), d_cnt.as<int32_t>(), nullptr, nullptr);
  API_CUDA(cudaGetLastError(), "brick counts");
  API_CUDA(exclusive_scan_i32(d_cnt.as<int32_t>(), g.nbricks, S.img_off.as<int64_t>(), d_scan.as<int64_t>(), st), "scan");
  API_CUDA(cudaMemcpyAsync(&g.nimg, S.img_off.as<int64_t>() + g.nbricks, sizeof(int64_t), cudaMemcpyDeviceToHost, st), "D2H");
  API_CUDA(cudaStreamSynchronize(st), "brick counts");
  if (g.nimg * P >= ((int64_t)1 << 31)) {
    *fits = false;
    return LCP_OK;
  }
  const int64_t ni = std::max<int64_t>(g.nimg, 1);
  API_CUDA(d_key.ensure(ni * sizeof(uint64_t)), "alloc");
  API_CUDA(d_per.ensure(ni * sizeof(int4)), "alloc");
  API_CUDA(S.img_atom.ensure(ni * sizeof(int32_t)), "alloc");
  API_CUDA(S.slot.ensure(ni * P * sizeof(int32_t)), "alloc");
  API_CUDA(d_row0.ensure(ni * sizeof(int32_t)), "alloc");
  API_CUDA(d_cc.ensure(g.nbricks * sizeof(int32_t)), "alloc");
  API_CUDA(cudaMemsetAsync(d_cnt.p, 0, g.nbricks * sizeof(int32_t), st), "memset");
  f64_images_kernel<true><<<bxs, 256, 0, st>>>(bg, dbx, no, d_flag.as<int32_t>(), d_cnt.as<int32_t>(),
                                               S.img_off.as<int64_t>(), d_key.as<uint64_t>());
  API_CUDA(cudaGetLastError(), "brick images");
  API_CUDA(d_tc.ensure(g.nbricks * sizeof(int32_t)), "alloc");
  f64_sort_kernel<<<blocks_for(g.nbricks * 32), 256, 0, st>>>(bg, dbx, no, g.nbricks, S.img_off.as<int64_t>(),
                                                              d_key.as<uint64_t>(), d_flag.as<int32_t>(),
                                                              S.img_atom.as<int32_t>(), d_per.as<int4>(),
                                                              d_row0.as<int32_t>(), d_cnt.as<int32_t>(),
                                                              d_cc.as<int32_t>(), d_tc.as<int32_t>());
  API_CUDA(cudaGetLastError(), "brick sort");
  API_CUDA(exclusive_scan_i32(d_cnt.as<int32_t>(), g.nbricks, d_row_off.as<int64_t>(), d_scan.as<int64_t>(), st), "scan");
  API_CUDA(exclusive_scan_i32(d_cc.as<int32_t>(), g.nbricks, d_chunk_off.as<int64_t>(), d_scan.as<int64_t>(), st), "scan");
  API_CUDA(exclusive_scan_i32(d_tc.as<int32_t>(), g.nbricks, d_tab_off.as<int64_t>(), d_scan.as<int64_t>(), st), "scan");
  int64_t ntab = 0;
  std::vector<int32_t> rows(g.nbricks);
  API_CUDA(cudaMemcpyAsync(&ntab, d_tab_off.as<int64_t>() + g.nbricks, sizeof(int64_t), cudaMemcpyDeviceToHost, st), "D2H");
  API_CUDA(cudaMemcpyAsync(&g.nrows, d_row_off.as<int64_t>() + g.nbricks, sizeof(int64_t), cudaMemcpyDeviceToHost, st), "D2H");
  API_CUDA(cudaMemcpyAsync(&g.nchunks, d_chunk_off.as<int64_t>() + g.nbricks, sizeof(int64_t), cudaMemcpyDeviceToHost, st), "D2H");
  API_CUDA(cudaMemcpyAsync(rows.data(), d_cnt.p, g.nbricks * sizeof(int32_t), cudaMemcpyDeviceToHost, st), "D2H");
  f64_fill_kernel<<<blocks_for(ni * P), 256, 0, st>>>(S.slot.as<int32_t>(), g.nimg * P, -1);
  API_CUDA(cudaGetLastError(), "brick slots");
  f64_slot_kernel<<<pts, 256, 0, st>>>(bg, dbx, no, d_flag.as<int32_t>(), S.slot.as<int32_t>());
  API_CUDA(cudaGetLastError(), "brick slots");
  API_CUDA(cudaStreamSynchronize(st), "brick rows");
  for (int32_t r : rows) g.max_rows = std::max(g.max_rows, r);
  if (g.max_rows > kF64MaxRows) *fits = false;
  if (ntab >= ((int64_t)1 << 32)) *fits = false;
  // a quarter of the device's memory stays free for what a program allocates
  // next: hundreds of cells whose orbital tables fit beside each other still do
  // (256 of them take 77 GB, and these tables would take 200)
  size_t mem_free = 0, mem_total = 0;
  API_CUDA(cudaMemGetInfo(&mem_free, &mem_total), "memory");
  const size_t need = (size_t)g.nchunks * 32 * P * sizeof(uint64_t) + mem_total / 4;
  if (*fits && mem_free < need) {
    S.release();
    S.need = need;
  }
  if (!*fits || S.need) return LCP_OK;
  API_CUDA(S.rows.ensure(std::max<int64_t>(g.nrows, 1) * sizeof(F64Row)), "alloc");
  API_CUDA(S.tab.ensure(std::max<int64_t>(ntab, 1) * sizeof(int32_t)), "alloc");
  API_CUDA(S.table.ensure(std::max<int64_t>(g.nchunks, 1) * 32 * P * sizeof(uint64_t)), "alloc");
  API_CUDA(S.bricks.ensure(g.nbricks * sizeof(F64Brick)), "alloc");
  f64_bricks_kernel<<<blocks_for(g.nbricks), 256, 0, st>>>(g.nbricks, S.img_off.as<int64_t>(), d_row_off.as<int64_t>(),
                                                           d_chunk_off.as<int64_t>(), d_tab_off.as<int64_t>(),
                                                           S.bricks.as<F64Brick>());
  API_CUDA(cudaGetLastError(), "bricks");
  g.bricks = S.bricks.as<F64Brick>();
  g.rows = S.rows.as<F64Row>();
  g.table = S.table.as<uint64_t>();
  g.tab = S.tab.as<int32_t>();
  if (P == 128) {
    API_CUDA(S.ptexp.ensure(g.nbricks * (P + 1) * sizeof(int32_t)), "alloc");  // and bad
    f64_fill_kernel<<<blocks_for(g.nbricks * P), 256, 0, st>>>(S.ptexp.as<int32_t>(), g.nbricks * P, 1);
    API_CUDA(cudaGetLastError(), "brick scales");
    g.ptexp = S.ptexp.as<int32_t>();
    g.bad = g.ptexp + g.nbricks * P;
    API_CUDA(cudaMemsetAsync(S.ptexp.as<int32_t>() + g.nbricks * P, 0, g.nbricks * sizeof(int32_t), st), "memset");
  } else {
    API_CUDA(S.cover.ensure(g.nbricks * sizeof(uint64_t)), "alloc");
    g.cover = S.cover.as<uint64_t>();
  }
  S.src = F64Source{o->phi.as<double>(), o->geom.phi_off, no, S.img_off.as<int64_t>(), S.img_atom.as<int32_t>(),
                    S.slot.as<int32_t>()};
  API_CUDA(launch_f64_table(g, S.src, d_row0.as<int32_t>(), S.rows.as<F64Row>(), S.ptexp.as<int32_t>(),
                            S.cover.as<uint64_t>(), S.table.as<uint64_t>(), st),
           "brick table");
  f64_tab_kernel<<<(unsigned)std::min<int64_t>(g.nbricks, 152 * 32), 256, 0, st>>>(
      o->f64_pairs, g.nbricks, S.img_off.as<int64_t>(), S.img_atom.as<int32_t>(), d_per.as<int4>(),
      d_tab_off.as<int64_t>(), P == 64 ? 1 : 0, S.tab.as<int32_t>());
  API_CUDA(cudaGetLastError(), "brick pairs");
  API_CUDA(cudaStreamSynchronize(st), "brick tables");  // before the scratch above is freed
  ctx->launches += 20;
  return LCP_OK;
}

}  // namespace
}  // namespace lcp

// Predicted device bytes of both tilings (their tables dominate).
int64_t f64_footprint_estimate(const lcp_orbs* o) {
  const lcp::UCell& u = o->ucell->u;
  double bytes = 0.0;
  for (int P : {64, 128}) {
    int32_t bd[3] = {1, 1, 1};
    const double rows = lcp::choose_shape(u, P, bd);
    double nb = 1.0;
    for (int d = 0; d < 3; ++d) nb *= (double)((u.ngrid[d] + bd[d] - 1) / bd[d]);
    double no = 0.0;
    for (int a = 0; a < u.natom; ++a) no += u.numorbs[a];
    const double images = rows * u.natom / std::max(no, 1.0);
    bytes += nb * ((rows + 16.0) * (P * 8.0 + 8.0) + images * (images + P + 1.0) * 4.0);
  }
  return (int64_t)bytes;
}

// ensure_f64 builds the tilings it is asked for (kF64Density, kF64Elements)
// once per orbital set.  Afterwards a tiling's state is 1, or -1 for a cell
// beyond the kernels' limits (block offsets of 30 bits, bricks of kF64MaxRows
// rows), which keeps the pair kernels.  Without room for its tables it stays 0, on
// the pair kernels, and is tried again once enough memory is free (asking for that
// takes 0.1 ms at most, a step with the pair kernels of such a cell ten or more).
namespace {
lcp_status pair_tables(lcp_ctx* ctx, lcp_orbs* o) {
  if (o->f64_pairs_ready) return LCP_OK;
  const lcp::UCell& u = o->ucell->u;
  cudaStream_t st = ctx->stream;
  std::vector<int64_t> boff(u.block_off.begin(), u.block_off.end()), first(u.natom + 1, 0);
  for (int32_t a : u.pair_atom) first[a + 1]++;
  for (int a = 0; a < u.natom; ++a) first[a + 1] += first[a];
  DBuf* q = o->f64_pair_buf;
  API_CUDA(upload(q[0], u.pair_atom, st), "upload");
  API_CUDA(upload(q[1], u.pair_jatom, st), "upload");
  API_CUDA(upload(q[2], u.pair_cell, st), "upload");
  API_CUDA(upload(q[3], u.partner, st), "upload");
  API_CUDA(upload(q[4], boff, st), "upload");
  API_CUDA(upload(q[5], first, st), "upload");
  API_CUDA(upload(q[6], u.atv_ijk, st), "upload");
  API_CUDA(upload(q[7], u.ratv, st), "upload");
  lcp::F64Pairs& p = o->f64_pairs;
  p.natom = u.natom;
  p.ncell = u.ncell;
  p.cpy = u.cpycell;
  p.npairs = u.nloop;
  p.atom = q[0].as<int32_t>();
  p.jatom = q[1].as<int32_t>();
  p.cell = q[2].as<int32_t>();
  p.partner = q[3].as<int32_t>();
  p.boff = q[4].as<int64_t>();
  p.first = q[5].as<int64_t>();
  p.ijk = q[6].as<int32_t>();
  p.ratv = q[7].as<int32_t>();
  p.numorbs = o->geom.numorbs;
  o->f64_pairs_ready = true;
  return LCP_OK;
}
}  // namespace

lcp_status ensure_f64(lcp_ctx* ctx, lcp_orbs* o, int which) {
  std::lock_guard<std::mutex> lock(o->f64_mutex);
  for (int k = 0; k < 2; ++k) {
    F64Set& S = k ? o->f64_elements : o->f64_density;
    if (!(which & (1 << k)) || S.state != 0 || ctx->no_optional) continue;
    size_t mem_free = 0, mem_total = 0;
    if (S.need) {
      API_CUDA(cudaMemGetInfo(&mem_free, &mem_total), "memory");
      if (mem_free < S.need) continue;
      S.need = 0;
    }
    const lcp::UCell& u = o->ucell->u;
    bool fits = u.total_hsize < ((int64_t)1 << 30) && u.natom <= 65535 && u.nloop > 0;
    if (fits) {
      lcp_status s = pair_tables(ctx, o);
      if (s == LCP_OK) s = lcp::build_set(ctx, o, o->f64_pair_buf[6], S, k ? 64 : 128, &fits);
      if (s == LCP_ENOMEM) {  // the pair kernels need none of it
        (void)cudaGetLastError();
        S.release();
        API_CUDA(cudaMemGetInfo(&mem_free, &mem_total), "memory");
        S.need = mem_free + ((size_t)1 << 28);
      } else if (s) {
        return s;
      }
    }
    if (!fits) S.release();
    if (!S.need) S.state = fits ? 1 : -1;
  }
  return LCP_OK;
}

// The context's workspace of the FP64 contractions on this orbital set;
// ready: only reports whether it is there.
lcp_status ensure_f64_workspace(lcp_ctx* ctx, const lcp_orbs* o, bool* ready) {
  const lcp::UCell& u = o->ucell->u;
  const size_t hs = (size_t)u.total_hsize, nb = (size_t)o->f64_elements.g.nbricks, nd = (size_t)o->f64_density.g.nbricks;
  const std::pair<DBuf*, size_t> need[] = {
      {&ctx->w_f64d, (hs * lcp::kF64Copies + 2) * sizeof(double)},  // symmetrised D, twice (density); the sums of H
      {&ctx->w_f64c, ((size_t)u.natom * 33 + lcp::kF64CmaxTail) * sizeof(uint32_t)},  // D's column maxima
      {&ctx->w_f64v, std::max<size_t>(nb, 1) * 64 * sizeof(int64_t)},  // V by brick
      {&ctx->w_f64e, std::max<size_t>(2 * std::max(nb, nd), 1) * sizeof(int32_t)}};  // its scales, or D's by brick (density), and odd bricks
  if (ready) {
    *ready = true;
    for (const auto& n : need) *ready = *ready && n.first->p && n.first->bytes >= n.second;
    return LCP_OK;
  }
  for (size_t i = 0; i < 4; ++i) {
    DBuf& b = *need[i].first;
    if (((ctx->f64_captured >> i) & 1u) && b.p && b.bytes < need[i].second) {
      ctx->kept.emplace_back();
      ctx->kept.back().swap(b);
      ctx->f64_captured &= ~(1u << i);
    }
    API_CUDA(b.ensure(need[i].second), "alloc");
  }
  return LCP_OK;
}
