// Ray generation, first-hit traversal and per-patch count reduction on sm_100a.
//
// Ray stream (generate_rays, porerad/view_factors.py:135-182): ray r of patch p in
// the block of seed s takes draws (p*R + r)*4 + c, c = 0..3, of that block's PCG64
// stream.  Each thread jumps its stream there with the power-of-two affine maps of
// the LCG, so rays are generated on the fly in any order and never stored.
//   c = 0, 1: origin offsets clip(u, 1e-12, 1 - 1e-12) - 0.5 along the two face
//             tangents, then y, z wrapped with NumPy's float remainder;
//   c = 2, 3: radius = sqrt(u2), azimuth = (2 pi) u3, cos(theta) = sqrt(1 - u2);
//             the direction is divided by sqrt((dx^2 + dy^2) + dz^2).
// Traversal (_trace_kernel, view_factors.py:202-258): Amanatides-Woo cell walk in
// binary64 with the 1e-12 tie tolerance, periodic y/z, exits through x < 0 (hot
// wall) or x >= nx (cold wall), step cap max(10 N^3 + 10, min(8 nx (1 + (|dy|+|dz|)
// /|dx|) + 100, 1e8)).  Every operation is an explicit round-to-nearest intrinsic,
// so the arithmetic is the reference's operation for operation.  The occupancy
// probe reads one bit of the packed grid (L1/L2 resident).
#include <cub/device/device_scan.cuh>

#include <map>
#include <mutex>
#include <tuple>

#include "pr_math.cuh"
#include "pr_objects.cuh"

namespace pr {

// Per-seed table of LCG jump maps (A, C): state -> A state + C.
//   [0, 128):   the maps of 2^i steps, i = 0..63
//   [128, 192): the maps of 4 l steps, l = 0..31 (lane offsets inside a batch of 32 rays)
//   [192, 194): the map of 128 steps (one batch of 32 rays)
static constexpr int kMapStride = 256;
static constexpr int kMapSmall = 128;
static constexpr int kMapBatch = 192;

#define PR_TIE 1.0e-12
#ifndef PR_FULL
#define PR_FULL 0xffffffffu
#endif
#define PR_FAR 1.0e300
#define PR_TWO_PI 0x1.921fb54442d18p+2  // the binary64 product 2.0 * numpy.pi

struct Geom {
  const uint32_t* __restrict__ occ;
  const int32_t* __restrict__ ftab;
  int32_t nx, ny, nz;
  int64_t n_cells;
};

struct RaySrc {
  const double* __restrict__ origin;  // (P, 3)
  const int8_t* __restrict__ code;    // emission normal 0..5
  const pr_u128* __restrict__ maps;   // per seed: kMapStride entries, see SeedTables
  const pr_u128* __restrict__ state;  // per seed
  const pr_u128* __restrict__ inc;    // per seed
  double ny_d, nz_d;
};

__device__ __forceinline__ double clip_edge(double u) {
  const double lo = 1.0e-12, hi = 1.0 - 1.0e-12;
  return u < lo ? lo : (u > hi ? hi : u);
}

// Offset clip(u) - 0.5 of an origin along a face tangent.
__device__ __forceinline__ double face_offset(double u) {
  const double t = pr_sub(u, 0.5);
  return fabs(t) < 0.499 ? t : pr_sub(clip_edge(u), 0.5);
}

// NumPy's float remainder by b > 0 for the origins, whose values lie in (-b, 2b):
// a - b is exact there (Sterbenz), a + b is the single rounded add NumPy makes for a
// negative fmod result, and a zero result is +0.0.  Other values take the general path.
__device__ __forceinline__ double wrap_origin(double a, double b) {
  if (a > 0.0 && a < b) return a;
  if (a > -b && a < 2.0 * b) {
    if (a >= b) return pr_sub(a, b);
    if (a < 0.0) return pr_add(a, b);
    return a == 0.0 ? 0.0 : a;
  }
  return pr_pymod_pos(a, b);
}

// Unit direction of a ray from its draws u2, u3 about the emission normal `code`
// (view_factors.py:160-181).  Tangent axes (first, second) of a normal along x, y, z: (y, z),
// (x, z), (x, y).
__device__ __forceinline__ void ray_direction(double u2, double u3, int code, double& dx, double& dy, double& dz) {
  const int ax = code >> 1;
  const double sign = (code & 1) ? -1.0 : 1.0;
  const double radius = pr_sqrt(u2);
  double sn, cs;
  pr_sincos_2pi(pr_mul(PR_TWO_PI, u3), &sn, &cs);
  const double la = pr_mul(radius, cs);
  const double lb = sign * pr_mul(radius, sn);
  const double dn = sign * pr_sqrt(pr_sub(1.0, u2));
  dx = ax == 0 ? dn : la;
  dy = ax == 0 ? la : (ax == 1 ? dn : lb);
  dz = ax == 2 ? dn : lb;
  pr_unit_vector(&dx, &dy, &dz);
}

// Origin of a ray of patch p from its draws u0, u1 (view_factors.py:148-159).
__device__ __forceinline__ void ray_origin(const double* __restrict__ origin, double ny_d, double nz_d, int code,
                                           int64_t p, double u0, double u1, double& ox, double& oy, double& oz) {
  const int ax = code >> 1;
  ox = origin[3 * p];
  oy = origin[3 * p + 1];
  oz = origin[3 * p + 2];
  const double ta = face_offset(u0), tb = face_offset(u1);
  if (ax != 0) ox = pr_add(ox, ta);
  if (ax != 1) oy = pr_add(oy, ax == 0 ? ta : tb);
  if (ax != 2) oz = pr_add(oz, tb);
  oy = wrap_origin(oy, ny_d);
  oz = wrap_origin(oz, nz_d);
}

// Origin and direction of a ray of patch p whose stream stands before its four draws.
__device__ __forceinline__ void ray_from_stream(const double* __restrict__ origin, const int8_t* __restrict__ codes,
                                                double ny_d, double nz_d, pr_u128 st, pr_u128 inc, int64_t p,
                                                double& ox, double& oy, double& oz, double& dx, double& dy,
                                                double& dz) {
  const double u0 = pr_pcg_next_double(&st, inc);
  const double u1 = pr_pcg_next_double(&st, inc);
  const double u2 = pr_pcg_next_double(&st, inc);
  const double u3 = pr_pcg_next_double(&st, inc);
  const int code = codes[p];
  ray_origin(origin, ny_d, nz_d, code, p, u0, u1, ox, oy, oz);
  ray_direction(u2, u3, code, dx, dy, dz);
}

// Ray r of patch p, block s, of a stream not yet positioned.
__device__ __forceinline__ void make_ray(const RaySrc& src, int64_t p, int64_t r, int64_t R, int s,
                                         double& ox, double& oy, double& oz, double& dx, double& dy, double& dz) {
  const pr_u128* maps = src.maps + (int64_t)s * kMapStride;
  const pr_u128 st = pr_pcg_jump(src.state[s], (uint64_t)((p * R + r) * 4), maps);
  ray_from_stream(src.origin, src.code, src.ny_d, src.nz_d, st, src.inc[s], p, ox, oy, oz, dx, dy, dz);
}

__device__ __forceinline__ int64_t first_cell(double pos, double dir) {
  int64_t idx = (int64_t)floor(pos);
  if (dir < 0.0 && fabs(pr_sub(pos, rint(pos))) <= PR_TIE) idx -= 1;
  return idx;
}

__device__ __forceinline__ void axis_setup(double pos, double dir, int64_t idx, int& step, double& tmax,
                                           double& tdel) {
  if (dir > 0.0) {
    step = 1;
    tmax = pr_div(pr_sub(pr_add((double)idx, 1.0), pos), dir);
    tdel = pr_div(1.0, dir);
  } else if (dir < 0.0) {
    step = -1;
    tmax = pr_div(pr_sub((double)idx, pos), dir);
    tdel = pr_div(-1.0, dir);
  } else {
    step = 0;
    tmax = PR_FAR;
    tdel = PR_FAR;
  }
}

__device__ __forceinline__ int64_t imod(int64_t a, int64_t n) {
  int64_t m = a % n;
  return m < 0 ? m + n : m;
}

// imod for a value given as a binary64 integer (a floor) and n < 2^31: 32-bit arithmetic when
// the value fits in 32 bits (every wrap of a ray's coordinate in practice), else imod.
__device__ __forceinline__ int imod_floor(double f, int n) {
  if (fabs(f) < 2147483647.0) {
    const int m = (int)f % n;
    return m < 0 ? m + n : m;
  }
  return (int)imod((int64_t)f, (int64_t)n);
}

// Hit code of the ray (its index into the face table: cell 6 + face, or 6 n_cells + (0 hot |
// ny nz cold) + j nz + k), or -1 when it meets none; *steps counts the cells visited.
__device__ int64_t dda_hit_code(const Geom& g, double ox, double oy, double oz, double dx, double dy,
                                double dz, int64_t* steps) {
  *steps = 0;
  if (dx == 0.0) return -1;
  int64_t i = first_cell(ox, dx);
  const int64_t j0 = first_cell(oy, dy), k0 = first_cell(oz, dz);
  int sx, sy, sz;
  double tx, ty, tz, ddx, ddy, ddz;
  axis_setup(ox, dx, i, sx, tx, ddx);
  axis_setup(oy, dy, j0, sy, ty, ddy);
  axis_setup(oz, dz, k0, sz, tz, ddz);
  int jj = (int)imod(j0, g.ny), kk = (int)imod(k0, g.nz);
  double t = 0.0;
  int face = -1;
  double scale = pr_add(pr_mul(pr_mul(8.0, (double)g.nx),
                               pr_add(1.0, pr_div(pr_add(fabs(dy), fabs(dz)), fabs(dx)))), 100.0);
  if (scale > 100000000.0) scale = 100000000.0;
  int64_t cap = 10 * g.n_cells + 10;
  if ((int64_t)scale > cap) cap = (int64_t)scale;
  int64_t it = 0;
  for (; it < cap; ++it) {
    if (i < 0 || i >= g.nx) {
      const int64_t wj = imod((int64_t)floor(pr_add(oy, pr_mul(dy, t))), g.ny);
      const int64_t wk = imod((int64_t)floor(pr_add(oz, pr_mul(dz, t))), g.nz);
      *steps = it + 1;
      return 6 * g.n_cells + (i < 0 ? 0 : (int64_t)g.ny * g.nz) + wj * g.nz + wk;
    }
    const int64_t row = i * g.ny + jj;
    const int64_t cell = row * g.nz + kk;
    const uint32_t word = __ldg(g.occ + (cell >> 5));
    if ((word >> (cell & 31)) & 1u) {
      *steps = it + 1;
      return face >= 0 ? cell * 6 + face : -1;
    }
    double tn = tx;
    if (ty < tn) tn = ty;
    if (tz < tn) tn = tz;
    const bool cx = fabs(pr_sub(tx, tn)) <= PR_TIE;
    const bool cy = fabs(pr_sub(ty, tn)) <= PR_TIE;
    const bool cz = fabs(pr_sub(tz, tn)) <= PR_TIE;
    if (cx) {
      i += sx;
      tx = pr_add(tx, ddx);
      face = sx > 0 ? 1 : 0;
    }
    if (cy) {
      jj += sy;
      if (jj == g.ny) jj = 0;
      else if (jj < 0) jj = g.ny - 1;
      ty = pr_add(ty, ddy);
      if (!cx) face = sy > 0 ? 3 : 2;
    }
    if (cz) {
      kk += sz;
      if (kk == g.nz) kk = 0;
      else if (kk < 0) kk = g.nz - 1;
      tz = pr_add(tz, ddz);
      if (!cx && !cy) face = sz > 0 ? 5 : 4;
    }
    t = tn;
  }
  *steps = it;
  return -1;
}

// First patch hit by the ray, or -1 when it resolves none (the reference's failed flag).
__device__ __forceinline__ int32_t dda_first_hit(const Geom& g, double ox, double oy, double oz, double dx, double dy,
                                                 double dz, int64_t* steps) {
  const int64_t code = dda_hit_code(g, ox, oy, oz, dx, dy, dz, steps);
  return code >= 0 ? __ldg(g.ftab + code) : -1;
}

__device__ __forceinline__ void block_add_i64(int64_t v, unsigned long long* target) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(target, (unsigned long long)v);
}

__global__ void k_generate(RaySrc src, int64_t p0, int64_t np, int64_t R, double* __restrict__ origins,
                           double* __restrict__ dirs) {
  const int64_t n = np * R;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    double ox, oy, oz, dx, dy, dz;
    make_ray(src, p0 + q / R, q % R, R, 0, ox, oy, oz, dx, dy, dz);
    origins[3 * q] = ox;
    origins[3 * q + 1] = oy;
    origins[3 * q + 2] = oz;
    dirs[3 * q] = dx;
    dirs[3 * q + 1] = dy;
    dirs[3 * q + 2] = dz;
  }
}

__global__ void __launch_bounds__(256) k_trace_given(Geom g, const double* __restrict__ origins,
                                                     const double* __restrict__ dirs, int64_t n,
                                                     int32_t* __restrict__ recv,
                                                     unsigned long long* __restrict__ counters) {
  int64_t my_steps = 0, my_fail = 0;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    int64_t st = 0;
    const int32_t hit = dda_first_hit(g, origins[3 * q], origins[3 * q + 1], origins[3 * q + 2], dirs[3 * q],
                                      dirs[3 * q + 1], dirs[3 * q + 2], &st);
    my_steps += st;
    my_fail += hit < 0;
    recv[q] = hit;
  }
  block_add_i64(my_steps, counters + 0);
  block_add_i64(my_fail, counters + 1);
}

// ---------------------------------------------------------------------------
// Pooled traversal.  A chunk of rays is numbered seed-major, g = (s * np + (p - p0)) * R + r,
// so inside one seed block consecutive rays are 4 draws apart in their PCG64 stream.  Each warp
// grabs units of consecutive rays from a global counter and generates them 32 at a time with all
// lanes converged (one 128-step map advances the batch base, one small map per lane); the rays'
// traversal states wait in a warp-private shared-memory pool until a lane is free.  Between
// refills every lane runs kRounds rounds of kLook cells.
//
// What bounds it is instruction issue, so a round holds nothing but the cell walk.
//  - It runs on a padded copy of the occupancy bits (pr_case::pad): x has layers of solid cells
//    outside the walls, so a wall is met as a solid cell, and y and z have a halo of kHalo periodic
//    copies, so no step tests for a wrap; the lanes' positions are moved back into the box only
//    every kHalo cells.  A cell is one linear index c that a crossing moves by plus or minus a
//    stride, and the face a ray enters a cell through follows from that change of c.
//  - The next axis is the one with the smallest high word of t (for positive numbers they order as
//    the numbers do, to 2^-20 of their size).  When the successive smallest words of a round differ
//    by two units or more, every crossing was of one axis alone, in order: the others were more
//    than 2^-20 of the power of two below t away, and that is more than PR_TIE while t >= 2^-19.
//    Else (a few in 10^4 steps) the round is walked again with the reference's comparisons in
//    binary64, where fl(t_a - tn) <= PR_TIE is t_a <= RD(tn + PR_TIE), t_a - tn being exact.
//  - Rays outside these premises (a first crossing before 2^-19, a zero direction component, a
//    start cell moved by the tie rule, a start outside the pores) are listed and walked by
//    dda_hit_code afterwards (k_trace_alone).
// All t are formed by dda_hit_code's additions in its order; the occupancy words of a round are
// loaded together, and the state past the first solid cell is dropped.  Finished rays are resolved,
// and the step cap is tested, at the refills only.  The hit codes written are 6 c + face in padded
// cells (walls: the x layer next to the box); the per-patch reduction maps them to patches with all
// lanes busy.  Nothing here calls a function that is not inlined: one call, however rare, cost 188
// bytes of spills around the walk at 80 registers (45.6 instead of 34.7 ms).
// Measured on the 128^3 foam at 1000 rays per patch (2.57e8 rays of 45 cells): 34.7 ms, where one
// round of four cells with wrap, wall and face tests in it took 60.0 ms; 101 instead of 205 warp
// instructions per ray, 0.6 issued per cycle and scheduler.
static constexpr int kWarps = 4;  // warps per block
static constexpr int kMaxCap = INT32_MAX - 64;  // step counts stay int32
static constexpr uint32_t kNoHit = 0xffffffffu;

struct WarpPool {
  // ready rays: t and delta t per axis, wall-exit data (o, d along y and z), (c, q, cap, signs)
  double2 txy[32], tzdx[32], dyz[32], exo[32], exd[32];
  int4 ids[32];
  // each lane's current ray: wall-exit data, (step cap, wave-wide index, signs)
  double2 lexo[32], lexd[32];
  int4 lid[32];
  // its walk while the warp generates rays, so that the generator has the registers
  double2 sxy[32], szdx[32], sdyz[32];
  int2 sc[32];
  // the generator (warp-uniform): rays [next, end) of chunk `chunk` by wave-wide ray index; the
  // stream of ray `next` of seed block `seed`, its patch, its index there, the block's rays left
  pr_u128 base;
  int next, end, chunk, seed, ray, left;
  int64_t patch;
  // of the chunk whose rays are in flight
  BoxMap box;
  int min_cap;
  double cap_dx;  // a direction with |dx| >= cap_dx has no larger step cap than min_cap
};

// One chunk of a launch: the rays of patches [p0, p0 + np) of one case, numbered seed-major
// inside the chunk (g = (s * np + p - p0) * R + r) and placed at global ray indices
// [start, start + n) of the launch, start a multiple of kAlign.  A launch (a wave) may hold
// chunks of many cases of different sizes.  Its rays' hit codes go to recv[start + g].
static constexpr int kAlign = 32;
struct WaveChunk {
  const uint32_t* occ;
  const uint32_t* pad;   // padded occupancy, or NULL (the launch then walks the flat one)
  const double* origin;
  const int8_t* code;
  const pr_u128* maps;   // kMapStride maps per seed of this case
  const pr_u128* state;  // per seed
  const pr_u128* inc;    // per seed
  int64_t n, np, p0, R, start, n_cells;
  BoxMap box;
  double ny_d, nz_d;
};

__device__ __forceinline__ int pad_div(int c, const PadDiv& d) { return (int)(__umulhi((unsigned)c, d.mul) >> d.shift); }

// v mod n for v in [-kHalo, n + kHalo]
__device__ __forceinline__ int wrap_halo(int v, int n) {
  v += v < 0 ? n : 0;
  v -= v >= n ? n : 0;
  if (n <= kHalo) {
    v %= n;
    v += v < 0 ? n : 0;
  }
  return v;
}

// Face-table index (cell_face_patch, then the hot and the cold wall's lattice sites) of a padded
// hit code.
__device__ __forceinline__ int64_t face_index(const BoxMap& B, uint32_t code) {
  const int at = (int)(code / 6u), face = (int)(code - 6u * (uint32_t)at);
  const int i = pad_div(at, B.plane), rem = at - i * B.plane.by;
  const int jp = pad_div(rem, B.row);
  const int j = wrap_halo(jp - kHalo, B.ny), k = wrap_halo(rem - jp * B.row.by - kHalo, B.nz), x = i - kPadX;
  const int64_t site = (int64_t)j * B.nz + k, lattice = (int64_t)B.ny * B.nz;
  if ((unsigned)x < (unsigned)B.nx) return (x * lattice + site) * 6 + face;
  return 6 * B.nx * lattice + (x < 0 ? 0 : lattice) + site;
}

// chunk holding global ray index u (chunks sorted by start)
__device__ __forceinline__ int find_chunk(const WaveChunk* __restrict__ chunks, int n_chunks, int64_t u) {
  int lo = 0, hi = n_chunks - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (chunks[mid].start <= u) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// t of the first crossing and the t between crossings of one axis (view_factors.py:189-199), cell
// the start cell floor(pos): (cell + 1 - pos) / dir or (cell - pos) / dir, and 1 / |dir|.  True when
// the ray has to be walked alone: t below 2^-19 (or not a number, for dir 0), or pos so near a cell
// boundary that the tie rule may move its cell.
__device__ __forceinline__ bool axis_start(double pos, double dir, int cell, double& t, double& dd) {
  const double ad = fabs(dir);
  const double c = __hiloint2double(0x43300000, cell) - 0x1.0p52;  // (double)cell, cell >= 0
  const double below = pr_sub(pos, c);
  dd = pr_rcp(ad);
  t = pr_div_rcp(dir > 0.0 ? pr_sub(pr_add(c, 1.0), pos) : below, ad, dd);
  return !(t >= 0x1.0p-19) || !(fabs(below - 0.5) < 0.5 - 2.0e-12);
}

// The next batch of rays of the unit in W (chunk C) into pool slots [0, cnt); returns cnt, 0 when
// the unit went on to another chunk or ended in a gap between chunks.
template <bool kFlat>
__device__ __forceinline__ int generate_batch(WarpPool& W, const WaveChunk* __restrict__ chunks, int n_chunks,
                                              int32_t* __restrict__ alone_list,
                                              unsigned long long* __restrict__ n_alone) {
  const int lane = threadIdx.x & 31;
  const int cur = W.chunk, next = W.next, end = W.end;
  const WaveChunk& C = chunks[cur];
  int left = W.left;
  if (left == 0) {
    // position the stream at ray `next` (a new unit, or the unit's next seed block or chunk)
    const int64_t g0 = (int64_t)next - C.start;
    if (g0 >= C.n) {
      __syncwarp();
      if (lane == 0) {
        const bool has = cur + 1 < n_chunks;
        W.chunk = has ? cur + 1 : cur;
        W.next = has ? min(end, (int)chunks[cur + 1].start) : end;
      }
      __syncwarp();
      return 0;
    }
    const int64_t npR = C.np * C.R;
    const int s0 = (int)(g0 / npR);
    const int64_t rem = g0 - (int64_t)s0 * npR;
    const pr_u128 st = pr_pcg_jump(C.state[s0], ((uint64_t)C.p0 * (uint64_t)C.R + (uint64_t)rem) * 4u,
                                   C.maps + (int64_t)s0 * kMapStride);
    left = (int)min(npR - rem, (int64_t)INT32_MAX);
    __syncwarp();
    if (lane == 0) {
      W.base = st;
      W.seed = s0;
      W.patch = C.p0 + rem / C.R;
      W.ray = (int)(rem % C.R);
    }
    __syncwarp();
  }
  const int cnt = min(32, min(left, end - next));
  const int s0 = W.seed;
  const pr_u128* maps = C.maps + (int64_t)s0 * kMapStride;
  const pr_u128 base = W.base;
  const int R = (int)C.R;
  const int64_t patch = W.patch;
  const int ray = W.ray;
  // The rays are made in three steps that hand their values on through the pool, so that each has
  // few of them in registers (lanes past cnt repeat the last patch and are not used).
  const int over = R >= 32 ? (ray + lane >= R) : (ray + lane) / R;
  const int64_t p = min(patch + over, C.p0 + C.np - 1);
  {
    pr_u128 st = pr_u128_affine(maps[kMapSmall + 2 * lane], maps[kMapSmall + 2 * lane + 1], base);
    const pr_u128 inc = C.inc[s0];
    const double u0 = pr_pcg_next_double(&st, inc);
    const double u1 = pr_pcg_next_double(&st, inc);
    W.exo[lane] = make_double2(u0, u1);
    const double u2 = pr_pcg_next_double(&st, inc);
    const double u3 = pr_pcg_next_double(&st, inc);
    W.exd[lane] = make_double2(u2, u3);
  }
  const int code = C.code[p];
  __syncwarp();
  {
    const double2 u = W.exd[lane];
    double dx, dy, dz;
    ray_direction(u.x, u.y, code, dx, dy, dz);
    W.exd[lane] = make_double2(dy, dz);
    W.txy[lane].x = dx;
  }
  __syncwarp();
  {
    const double2 u = W.exo[lane], d = W.exd[lane];
    const double dx = W.txy[lane].x, dy = d.x, dz = d.y;
    double ox, oy, oz;
    ray_origin(C.origin, C.ny_d, C.nz_d, code, p, u.x, u.y, ox, oy, oz);
    // DDA setup (view_factors.py:213-224); a direction of 0 gives a t that is not >= 2^-19
    const int ci = __double2int_rd(ox), cj = __double2int_rd(oy), ck = __double2int_rd(oz);
    double a, b, e, da, db, de;
    bool alone = axis_start(ox, dx, ci, a, da);
    alone |= axis_start(oy, dy, cj, b, db);
    alone |= axis_start(oz, dz, ck, e, de);
    alone |= (unsigned)ci >= (unsigned)W.box.nx || (unsigned)cj >= (unsigned)W.box.ny || (unsigned)ck >= (unsigned)W.box.nz;
    int qq = next + lane, cap = W.min_cap;
    const int c = kFlat ? (ci * W.box.ny + cj) * W.box.nz + ck
                        : (ci + kPadX) * W.box.plane.by + (cj + kHalo) * W.box.row.by + ck + kHalo;
    if (!alone) {
      alone = (__ldg((kFlat ? C.occ : C.pad) + ((unsigned)c >> 5)) >> (c & 31)) & 1u;
      if (fabs(dx) < W.cap_dx) {
        // step cap max(10 n_cells + 10, (int)min(8 nx (1 + (|dy| + |dz|) / |dx|) + 100, 1e8)), where the
        // second can be the larger
        double scale = pr_add(pr_mul(pr_mul(8.0, (double)W.box.nx),
                                     pr_add(1.0, pr_div(pr_add(fabs(dy), fabs(dz)), fabs(dx)))), 100.0);
        if (scale > 100000000.0) scale = 100000000.0;
        cap = max(cap, (int)scale);
      }
    }
    if (alone && lane < cnt) {
      alone_list[atomicAdd(n_alone, 1ull)] = qq;
      qq = -1;
    }
    W.txy[lane] = make_double2(a, b);
    W.tzdx[lane] = make_double2(e, da);
    W.dyz[lane] = make_double2(db, de);
    W.exo[lane] = make_double2(oy, oz);
    // q is the wave-wide ray index (< 2^31)
    W.ids[lane] = make_int4(c, qq, cap, (dx < 0.0 ? 1 : 0) | (dy < 0.0 ? 2 : 0) | (dz < 0.0 ? 4 : 0));
  }
  __syncwarp();
  if (lane == 0) {
    // the generator moves on by the batch
    W.base = pr_u128_affine(maps[kMapBatch], maps[kMapBatch + 1], base);
    const int over = R >= 32 ? (ray + cnt >= R) : (ray + cnt) / R;
    W.patch = patch + over;
    W.ray = ray + cnt - over * R;
    W.next = next + cnt;
    W.left = left - cnt;
  }
  __syncwarp();
  return cnt;
}

// floor(v) mod n of a wall coordinate.
__device__ __forceinline__ int wall_site(double v, int n) {
  const double f = floor(v);
  if (f >= 0.0 && f < (double)n) return (int)f;
  return imod_floor(f, n);
}

// One crossing of the axis with the smallest high word of t (x before y before z); gap keeps the
// smallest difference of successive ones.  An axis left out for a tie, or for a t within two units,
// is the next smallest, so it shows as a gap below two.
__device__ __forceinline__ void cross(double& tx, double& ty, double& tz, double ddx, double ddy, double ddz, int& c,
                                      int sx, int sy, int sz, int& last, int& gap) {
  const int hx = __double2hiint(tx), hy = __double2hiint(ty), hz = __double2hiint(tz);
  const int m = __vimin3_s32(hx, hy, hz);
  gap = min(gap, m - last);
  last = m;
  const bool px = hx == m, py = hy == m;
  c += px ? sx : (py ? sy : sz);
  if (px) tx = pr_add(tx, ddx);
  else if (py) ty = pr_add(ty, ddy);
  else tz = pr_add(tz, ddz);
}

// Cell (i, j, k) of a flat index.
__device__ __forceinline__ void flat_cell(const BoxMap& B, int c, int& i, int& j, int& k) {
  const int row = c / B.nz;
  k = c - row * B.nz;
  i = row / B.ny;
  j = row - i * B.ny;
}

// kFlat: the same pool over boxes without a padded occupancy (long ones a few cells wide, and thin ones of
// more cells than the padded codes hold).  Positions are (i, j, k), every crossing is the reference's with
// its ties, wraps and wall test, kLook cells are crossed before their occupancy is loaded, and the hit
// codes are face-table indices.  Instructions bound it, like the padded walk.  Four rounds of two cells, 6
// blocks per SM, the whole count pass: 200000 x 8 x 8 cells, 4.4e8 rays of 11 cells, 42.2 ms (rounds of
// three cells 42.7, four 42.5, one 45.2; one ray per thread 300; the pool before the padded walk 53.8);
// 250000 x 2 x 2, 3.8e6 rays of 101 cells, 9.0 (10.1, 9.1, 11.5; 13.5; 10.4); 4 x 4000 x 4000, 2.4e8 rays of
// 7, 56.8 (57.1, 57.3, 58.6; 200; 62.9).
template <int kMinBlocks, int kRounds, int kLook, bool kFlat>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) k_trace_pool(const WaveChunk* __restrict__ chunks,
                                                                        int n_chunks, int total, int max_unit,
                                                                        uint32_t* __restrict__ recv,
                                                                        int32_t* __restrict__ alone_list,
                                                                        unsigned long long* __restrict__ work,
                                                                        unsigned long long* __restrict__ chunk_ctr) {
  static_assert(kFlat || (kLook <= kPadX && kRounds * kLook <= kHalo), "a round stays inside the padded grid");
  constexpr int kSettle = kFlat ? 1 : kHalo / (kRounds * kLook);  // refills between moves back into the box
  __shared__ WarpPool pools[kWarps];
  WarpPool& W = pools[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;

  int cur = -1;                     // warp-uniform: the chunk of the rays in flight
  const uint32_t* occ = nullptr;    // its occupancy, padded or flat
  int head = 0, tail = 0;           // warp-uniform: the pool holds slots [head, tail)
  int settle = 0;
  bool more = true;                 // warp-uniform
  if (lane == 0) W.next = W.end = 0;
  __syncwarp();

  // state: 0 no ray, 1 walking; 2 and 3 in its solid cell c, entered from cell `from` of its last
  // round at t = te (3), or te is the tx that round began with in cell `begin` (2); flat: met the face
  // with code `from` (2), or left through the hot (from = 0) or cold (1) wall at t = te (3)
  int state = 0, c = 0, sx = 0, sy = 0, sz = 0, it = 0, from = 0, begin = 0;
  int i = 0, j = 0, k = 0;  // flat: the cell
  double tx = 0, ty = 0, tz = 0, ddx = 0, ddy = 0, ddz = 0, te = 0;
  unsigned my_steps = 0;

  for (;;) {
    // ---- finished rays: hit code, step cap
    if (state != 0) {
      const bool capped = it >= W.min_cap;
      if (state >= 2 || capped) {
        uint32_t hit = kNoHit;
        bool done = state >= 2;
        if (done && kFlat) {
          hit = (uint32_t)from;
          if (state == 3) {
            const int ny = W.box.ny, nz = W.box.nz;
            const double2 o = W.lexo[lane], d = W.lexd[lane];
            const int wj = wall_site(pr_add(o.x, pr_mul(d.x, te)), ny), wk = wall_site(pr_add(o.y, pr_mul(d.y, te)), nz);
            hit = (uint32_t)((6 * W.box.nx + from) * ny * nz + wj * nz + wk);
          }
        } else if (done) {
          const int low = kPadX * W.box.plane.by, high = low + W.box.nx * W.box.plane.by;
          if (c < low || c >= high) {
            // a wall: the x layer next to the box at the exit position (view_factors.py:226-229); a
            // round without ties crossed x alone, the last time at tx after the crossings before
            const int layer = c < low ? kPadX - 1 : kPadX + W.box.nx;
            if (state == 2)
              for (int h = abs(layer - pad_div(begin, W.box.plane)); h > 1; --h) te = pr_add(te, ddx);
            const double2 o = W.lexo[lane], d = W.lexd[lane];
            const int wj = wall_site(pr_add(o.x, pr_mul(d.x, te)), W.box.ny);
            const int wk = wall_site(pr_add(o.y, pr_mul(d.y, te)), W.box.nz);
            hit = 6u * (uint32_t)(layer * W.box.plane.by + (wj + kHalo) * W.box.row.by + wk + kHalo);
          } else {
            // the face: x if x was crossed, else y, else z; 0..5 = +x, -x, +y, -y, +z, -z of the
            // solid cell, so the first of each pair is entered moving down
            const int move = c - from, far = 2 * abs(move);
            const int axis = far > W.box.plane.by ? 0 : (far > W.box.row.by ? 2 : 4);
            hit = 6u * (uint32_t)c + (uint32_t)(axis + (move > 0 ? 1 : 0));
          }
        }
        const int4 id = W.lid[lane];
        if (capped && it + (done ? 0 : 1) > id.x) {
          done = true;
          hit = kNoHit;
          it = id.x;
          atomicAdd(chunk_ctr + 2 * cur + 1, 1ull);
        }
        if (done) {
          recv[id.y] = hit;  // no load on this path: the RLE pass maps codes to patches
          my_steps += (unsigned)it;
          if (my_steps >= 0x40000000u) {
            atomicAdd(chunk_ctr + 2 * cur, (unsigned long long)my_steps);
            my_steps = 0;
          }
          state = 0;
        }
      }
    }
    // ---- free lanes take ready rays; an empty pool is refilled with the next batch of 32
    unsigned idle = __ballot_sync(PR_FULL, state == 0);
    while (idle) {
      if (head < tail) {
        const int avail = tail - head;
        if (state == 0) {
          const int rank = __popc(idle & ((1u << lane) - 1u));
          if (rank < avail) {
            const int slot = head + rank;
            const int4 id = W.ids[slot];
            const double2 a = W.txy[slot], b = W.tzdx[slot], e = W.dyz[slot];
            W.lexo[lane] = W.exo[slot];
            W.lexd[lane] = W.exd[slot];
            W.lid[lane] = make_int4(id.z, id.y, id.w, 0);
            tx = a.x; ty = a.y; tz = b.x;
            ddx = b.y; ddy = e.x; ddz = e.y;
            c = id.x;
            sx = kFlat ? 1 : W.box.plane.by;
            sy = kFlat ? 1 : W.box.row.by;
            if (id.w & 1) sx = -sx;
            if (id.w & 2) sy = -sy;
            sz = (id.w & 4) ? -1 : 1;
            if constexpr (kFlat) flat_cell(W.box, c, i, j, k);
            it = 1;  // the start cell
            state = id.y >= 0;  // a ray already walked alone leaves a slot with q = -1
          }
        }
        head += min(__popc(idle), avail);
        __syncwarp();
        idle = __ballot_sync(PR_FULL, state == 0);
        continue;
      }
      if (!more) break;
      const int next = W.next;
      if (next >= W.end) {
        // a new unit; units shrink with the rays left, so that the warps end together
        const int unit = max(32, min(max_unit, (total - next) / (int)(gridDim.x * kWarps * 4) & ~31));
        unsigned long long u = 0;
        if (lane == 0) u = atomicAdd(work, (unsigned long long)unit);
        u = __shfl_sync(PR_FULL, u, 0);
        if (u >= (unsigned long long)total) {
          more = false;
          break;
        }
        if (lane == 0) {
          W.chunk = find_chunk(chunks, n_chunks, (int64_t)u);
          W.next = (int)u;
          W.end = min((int)u + unit, total);
          W.left = 0;
        }
        __syncwarp();
      }
      if (W.chunk != cur) {
        // another chunk's rays wait until nothing of this one is in flight
        if (idle != PR_FULL) break;
        if (cur >= 0 && my_steps) atomicAdd(chunk_ctr + 2 * cur, (unsigned long long)my_steps);
        my_steps = 0;
        cur = W.chunk;
        __syncwarp();
        if (lane == 0) {
          W.box = chunks[cur].box;
          const int cap = (int)min((int64_t)kMaxCap, 10 * chunks[cur].n_cells + 10);
          W.min_cap = cap;
          // |dy| + |dz| <= sqrt 2, so 8 nx (1 + (|dy| + |dz|) / |dx|) + 100 <= cap from this |dx| on
          const double first = 8.0 * W.box.nx, room = (double)cap - 101.0 - first;
          W.cap_dx = room > 0.0 ? 1.4143 * first / room : 2.0;
        }
        __syncwarp();
      }
      W.sxy[lane] = make_double2(tx, ty);
      W.szdx[lane] = make_double2(tz, ddx);
      W.sdyz[lane] = make_double2(ddy, ddz);
      W.sc[lane] = make_int2(kFlat ? (i * W.box.ny + j) * W.box.nz + k : c, it);
      __syncwarp();
      head = 0;
      tail = generate_batch<kFlat>(W, chunks, n_chunks, alone_list, work + 1);
      __syncwarp();
      {
        const double2 a = W.sxy[lane], b = W.szdx[lane], e = W.sdyz[lane];
        const int2 v = W.sc[lane];
        tx = a.x; ty = a.y; tz = b.x;
        ddx = b.y; ddy = e.x; ddz = e.y;
        c = v.x;
        it = v.y;
        const int sign = W.lid[lane].z;
        sx = kFlat ? 1 : W.box.plane.by;
        sy = kFlat ? 1 : W.box.row.by;
        if (sign & 1) sx = -sx;
        if (sign & 2) sy = -sy;
        sz = (sign & 4) ? -1 : 1;
        if constexpr (kFlat) flat_cell(W.box, c, i, j, k);
        occ = kFlat ? chunks[cur].occ : chunks[cur].pad;
      }
    }
    if (idle == PR_FULL && !more) break;
    // ---- positions back into the box, y and z periodic
    if (settle == 0) {
      if (!kFlat && state == 1) {
        const int i = pad_div(c, W.box.plane), rem = c - i * W.box.plane.by;
        const int j = pad_div(rem, W.box.row), k = rem - j * W.box.row.by;
        const int ny = W.box.ny, nz = W.box.nz, by = W.box.row.by;
        c += (wrap_halo(j - kHalo, ny) - (j - kHalo)) * by + wrap_halo(k - kHalo, nz) - (k - kHalo);
      }
      settle = kSettle;
    }
    --settle;
    // ---- kRounds rounds of kLook cells (view_factors.py:225-255)
#pragma unroll 1
    for (int b = 0; b < kRounds; ++b) {
      if (state != 1) continue;
      if constexpr (kFlat) {
        const int nx = W.box.nx, ny = W.box.ny, nz = W.box.nz;
        int code[kLook], m = 0;  // the hit codes of the first m cells entered
        double tn = 0.0;
#pragma unroll
        for (int p = 0; p < kLook; ++p) {
          code[p] = 0;
          if (m < p) continue;  // through a wall
          tn = tx;
          if (ty < tn) tn = ty;
          if (tz < tn) tn = tz;
          const double lim = __dadd_rd(tn, PR_TIE);
          int face = 0;
          if (tz <= lim) {
            tz = pr_add(tz, ddz);
            k += sz;
            k = k == nz ? 0 : (k < 0 ? nz - 1 : k);
            face = sz > 0 ? 5 : 4;
          }
          if (ty <= lim) {
            ty = pr_add(ty, ddy);
            j += sy;
            j = j == ny ? 0 : (j < 0 ? ny - 1 : j);
            face = sy > 0 ? 3 : 2;
          }
          if (tx <= lim) {
            tx = pr_add(tx, ddx);
            i += sx;
            face = sx > 0 ? 1 : 0;
          }
          if ((unsigned)i < (unsigned)nx) {
            code[p] = ((i * ny + j) * nz + k) * 6 + face;
            m = p + 1;
          }
        }
        uint32_t bit[kLook];
#pragma unroll
        for (int p = 0; p < kLook; ++p) {
          const unsigned cell = (unsigned)code[p] / 6u;
          bit[p] = p < m ? __ldg(occ + (cell >> 5)) >> (cell & 31u) : 0u;
        }
        int used = m;
        if (m < kLook) {
          used = m + 1;
          state = 3;
          te = tn;
          from = i < 0 ? 0 : 1;
        }
#pragma unroll
        for (int p = kLook - 1; p >= 0; --p) {
          if (bit[p] & 1u) {
            used = p + 1;
            state = 2;
            from = code[p];
          }
        }
        it += used;
        continue;
      }
      const int c0 = c;
      const double x0 = tx, y0 = ty, z0 = tz;
      int cell[kLook], last = -4, gap = 4;
#pragma unroll
      for (int p = 0; p < kLook; ++p) {
        cross(tx, ty, tz, ddx, ddy, ddz, c, sx, sy, sz, last, gap);
        cell[p] = c;
      }
      gap = min(gap, __vimin3_s32(__double2hiint(tx), __double2hiint(ty), __double2hiint(tz)) - last);
      if (gap < 2) {
        // the same cells with the reference's tie rule, one at a time
        tx = x0;
        ty = y0;
        tz = z0;
        c = c0;
        for (int p = 0; p < kLook && state == 1; ++p) {
          double m = tx;
          if (ty < m) m = ty;
          if (tz < m) m = tz;
          const double lim = __dadd_rd(m, PR_TIE);
          from = c;
          if (tx <= lim) {
            tx = pr_add(tx, ddx);
            c += sx;
          }
          if (ty <= lim) {
            ty = pr_add(ty, ddy);
            c += sy;
          }
          if (tz <= lim) {
            tz = pr_add(tz, ddz);
            c += sz;
          }
          ++it;
          if ((__ldg(occ + ((unsigned)c >> 5)) >> (c & 31)) & 1u) {
            te = m;
            state = 3;
          }
        }
        continue;
      }
      uint32_t bit[kLook], any = 0;
#pragma unroll
      for (int p = 0; p < kLook; ++p) bit[p] = __ldg(occ + ((unsigned)cell[p] >> 5));
#pragma unroll
      for (int p = 0; p < kLook; ++p) {
        bit[p] = __funnelshift_r(bit[p], 0u, (unsigned)cell[p]);  // shift by cell mod 32
        any |= bit[p];
      }
      if (any & 1u) {
        // the first solid cell of the round
        c = cell[kLook - 1];
        from = cell[kLook - 2];
        int pos = kLook;
#pragma unroll
        for (int p = kLook - 2; p >= 0; --p) {
          if (bit[p] & 1u) {
            c = cell[p];
            from = p > 0 ? cell[p - 1] : c0;
            pos = p + 1;
          }
        }
        it += pos;
        begin = c0;
        te = x0;
        state = 2;
      } else {
        it += kLook;
      }
    }
  }
  if (cur >= 0 && my_steps) atomicAdd(chunk_ctr + 2 * cur, (unsigned long long)my_steps);
}

// One thread per ray: the rays of alone_list (work[1] of them), which the pooled walk leaves out.  Their hit
// codes are face-table indices where the case has no padded occupancy.
__global__ void __launch_bounds__(128) k_trace_alone(const WaveChunk* __restrict__ chunks, int n_chunks,
                                                     uint32_t* __restrict__ recv,
                                                     const int32_t* __restrict__ alone_list,
                                                     const unsigned long long* __restrict__ work,
                                                     unsigned long long* __restrict__ chunk_ctr) {
  const int n = (int)work[1];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int u = alone_list[e];
    const int cur = find_chunk(chunks, n_chunks, u);
    const WaveChunk& C = chunks[cur];
    const int64_t g0 = u - C.start, npR = C.np * C.R;
    const int s0 = (int)(g0 / npR);
    const int64_t rem = g0 - (int64_t)s0 * npR;
    const pr_u128 st = pr_pcg_jump(C.state[s0], ((uint64_t)C.p0 * (uint64_t)C.R + (uint64_t)rem) * 4u,
                                   C.maps + (int64_t)s0 * kMapStride);
    double ox, oy, oz, dx, dy, dz;
    ray_from_stream(C.origin, C.code, C.ny_d, C.nz_d, st, C.inc[s0], C.p0 + rem / C.R, ox, oy, oz, dx, dy, dz);
    Geom g;
    g.occ = C.occ;
    g.ftab = nullptr;
    g.nx = C.box.nx;
    g.ny = C.box.ny;
    g.nz = C.box.nz;
    g.n_cells = C.n_cells;
    int64_t steps;
    const int64_t hit = dda_hit_code(g, ox, oy, oz, dx, dy, dz, &steps);
    uint32_t code = kNoHit;
    if (hit >= 0 && !C.pad) {
      code = (uint32_t)hit;
    } else if (hit >= 0) {
      const int64_t wall = hit - 6 * g.n_cells, lattice = (int64_t)g.ny * g.nz;
      const int64_t cell = wall < 0 ? hit / 6 : wall % lattice;
      const int i = wall < 0 ? (int)(cell / lattice) : (wall < lattice ? -1 : g.nx);
      const int site = (int)(cell % lattice);
      code = 6u * (uint32_t)((i + kPadX) * C.box.plane.by + (site / g.nz + kHalo) * C.box.row.by + site % g.nz + kHalo) +
             (wall < 0 ? (uint32_t)(hit % 6) : 0u);
    }
    recv[u] = code;
    atomicAdd(chunk_ctr + 2 * cur, (unsigned long long)steps);
    if (hit < 0) atomicAdd(chunk_ctr + 2 * cur + 1, 1ull);
  }
}

// Per origin patch: gather its L = S * R receivers (seed-major chunk layout), sort them
// in shared memory (bitonic), run-length encode into (receiver, count) pairs at
// out[(p - p0) * L ...], nnz[p - p0].
struct RleChunk {
  const uint32_t* recv;  // hit codes of the chunk (seed-major)
  const int32_t* ftab;   // face table of its case
  BoxMap box;            // maps hit codes to it
  unsigned long long* fail;  // the chunk's failed-ray counter
  int64_t np;           // patches
  int64_t patch0;       // index of its first patch among the wave's patches
  int64_t ray0;         // offset of its rays (and stage entries) in the wave's buffers
};

// Receiving patch of a hit code, -1 for an unresolved ray; bad counts faces without a patch.
__device__ __forceinline__ int32_t receiver_of(const RleChunk& K, uint32_t code, int& bad) {
  if (code == kNoHit) return -1;
  const int32_t r = __ldg(K.ftab + (K.box.padded ? face_index(K.box, code) : (int64_t)code));
  bad += r < 0;
  return r;
}

__global__ void __launch_bounds__(512) k_patch_rle(const RleChunk* __restrict__ rc, int n_chunks,
                                                   int64_t total_patches, int L, int R, int Lpad,
                                                   int32_t* __restrict__ st_col, int32_t* __restrict__ st_cnt,
                                                   int32_t* __restrict__ nnz) {
  extern __shared__ int32_t sm[];
  int32_t* key = sm;          // Lpad
  int32_t* head = sm + Lpad;  // Lpad (positions of run heads)
  __shared__ int32_t warp_tot[16];
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int64_t gp = blockIdx.x; gp < total_patches; gp += gridDim.x) {
    int c = 0;
    {
      int lo = 0, hi = n_chunks - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (rc[mid].patch0 <= gp) lo = mid;
        else hi = mid - 1;
      }
      c = lo;
    }
    const int64_t p = gp - rc[c].patch0, np = rc[c].np;
    const RleChunk K = rc[c];
    for (int i = tid; i < Lpad; i += nt) {
      if (i < L) {
        const int sd = i / R;
        int bad = 0;
        key[i] = receiver_of(K, K.recv[((int64_t)sd * np + p) * R + (i - sd * R)], bad);
        if (bad) atomicAdd(K.fail, 1ull);
      } else {
        key[i] = INT32_MAX;
      }
    }
    __syncthreads();
    for (int k = 2; k <= Lpad; k <<= 1) {
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int t = tid; t < (Lpad >> 1); t += nt) {
          const int a = ((t / j) * 2 * j) + (t % j);
          const int b = a + j;
          const bool up = (a & k) == 0;
          const int32_t x = key[a], y = key[b];
          if ((x > y) == up) {
            key[a] = y;
            key[b] = x;
          }
        }
        __syncthreads();
      }
    }
    // heads: contiguous chunk per thread, then a block-wide exclusive scan
    const int per = (L + nt - 1) / nt;
    const int lo = tid * per, hi = min(L, lo + per);
    int mine = 0;
    for (int i = lo; i < hi; ++i) mine += (i == 0 || key[i] != key[i - 1]);
    int incl = mine;
    const int lane = tid & 31, wid = tid >> 5;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    int base = 0, total = 0;
    for (int w = 0; w < (nt >> 5); ++w) {
      if (w < wid) base += warp_tot[w];
      total += warp_tot[w];
    }
    int u = base + incl - mine;
    for (int i = lo; i < hi; ++i)
      if (i == 0 || key[i] != key[i - 1]) head[u++] = i;
    __syncthreads();
    int32_t* oc = st_col + rc[c].ray0 + p * L;
    int32_t* on = st_cnt + rc[c].ray0 + p * L;
    for (int v = tid; v < total; v += nt) {
      const int h = head[v];
      const int e = v + 1 < total ? head[v + 1] : L;
      oc[v] = key[h];
      on[v] = e - h;
    }
    if (tid == 0) nnz[gp] = total;
    __syncthreads();
  }
}

// The same reduction with one warp per origin patch, for Lpad = 32 K <= 1024: the patch's
// keys sit in registers, element e = r * 32 + lane in register r of lane `lane`, and are
// sorted by the bitonic network (partners e ^ j: across lanes by shuffles for j < 32,
// across registers for j >= 32); run heads and tails come from neighbour shuffles and
// ballots, head positions go through the warp's shared row, and every tail writes its
// (receiver, count).  Output layout as k_patch_rle.
template <int K>
__global__ void __launch_bounds__(128) k_patch_rle_warp(const RleChunk* __restrict__ rc, int n_chunks,
                                                        int64_t total_patches, int L, int R,
                                                        int32_t* __restrict__ st_col, int32_t* __restrict__ st_cnt,
                                                        int32_t* __restrict__ nnz) {
  constexpr int N = 32 * K;
  __shared__ int32_t heads[4][N];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t gp = blockIdx.x * (int64_t)(blockDim.x >> 5) + wid; gp < total_patches; gp += warps) {
    int c = 0;
    {
      int lo = 0, hi = n_chunks - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (rc[mid].patch0 <= gp) lo = mid;
        else hi = mid - 1;
      }
      c = lo;
    }
    const int64_t p = gp - rc[c].patch0, np = rc[c].np;
    const RleChunk chunk = rc[c];
    int32_t x[K];
    int bad = 0;
#pragma unroll
    for (int r = 0; r < K; ++r) {
      const int e = r * 32 + lane;
      int32_t v = INT32_MAX;
      if (e < L) {
        const int sd = e / R;
        v = receiver_of(chunk, chunk.recv[((int64_t)sd * np + p) * R + (e - sd * R)], bad);
      }
      x[r] = v;
    }
    if (bad) atomicAdd(rc[c].fail, (unsigned long long)bad);
    // bitonic sort, ascending
#pragma unroll
    for (int k = 2; k <= N; k <<= 1) {
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        if (j >= 32) {
          const int jr = j >> 5;
#pragma unroll
          for (int r = 0; r < K; ++r) {
            if ((r & jr) == 0) {
              const bool up = ((r * 32) & k) == 0;  // k >= 64 here: bit of r
              const int32_t a = x[r], b = x[r | jr];
              const bool sw = up ? (a > b) : (a < b);
              x[r] = sw ? b : a;
              x[r | jr] = sw ? a : b;
            }
          }
        } else {
          const bool lower = (lane & j) == 0;
#pragma unroll
          for (int r = 0; r < K; ++r) {
            const bool up = (k < 32 ? (lane & k) : ((r * 32) & k)) == 0;
            const int32_t y = __shfl_xor_sync(PR_FULL, x[r], j);
            const int32_t lo_v = min(x[r], y), hi_v = max(x[r], y);
            x[r] = (lower == up) ? lo_v : hi_v;
          }
        }
      }
    }
    // run heads (key differs from its predecessor) and tails (differs from its successor)
    int32_t* hrow = heads[wid];
    int base = 0;
#pragma unroll
    for (int r = 0; r < K; ++r) {
      const int e = r * 32 + lane;
      int32_t prev = __shfl_up_sync(PR_FULL, x[r], 1);
      const int32_t last_prev = __shfl_sync(PR_FULL, x[r > 0 ? r - 1 : 0], 31);
      if (lane == 0) prev = last_prev;
      const bool head = e < L && (e == 0 || x[r] != prev);
      const unsigned hb = __ballot_sync(PR_FULL, head);
      if (head) hrow[base + __popc(hb & lt)] = e;
      base += __popc(hb);
    }
    __syncwarp();
    int32_t* oc = st_col + rc[c].ray0 + p * L;
    int32_t* on = st_cnt + rc[c].ray0 + p * L;
    int runs = 0;  // heads at positions < e
#pragma unroll
    for (int r = 0; r < K; ++r) {
      const int e = r * 32 + lane;
      int32_t prev = __shfl_up_sync(PR_FULL, x[r], 1);
      const int32_t last_prev = __shfl_sync(PR_FULL, x[r > 0 ? r - 1 : 0], 31);
      if (lane == 0) prev = last_prev;
      int32_t next = __shfl_down_sync(PR_FULL, x[r], 1);
      const int32_t first_next = __shfl_sync(PR_FULL, x[r + 1 < K ? r + 1 : r], 0);
      if (lane == 31) next = first_next;
      const bool head = e < L && (e == 0 || x[r] != prev);
      const bool tail = e < L && (e == L - 1 || x[r] != next);
      const unsigned hb = __ballot_sync(PR_FULL, head);
      const int run = runs + __popc(hb & lt) + (head ? 1 : 0) - 1;  // run index of element e
      if (tail) {
        oc[run] = x[r];
        on[run] = e - hrow[run] + 1;
      }
      runs += __popc(hb);
    }
    if (lane == 0) nnz[gp] = base;
    __syncwarp();
  }
}

// Copy each row's unique pairs from the stage to its CSR position (warp per row).
__global__ void k_compact_rows(const int32_t* __restrict__ st_col, const int32_t* __restrict__ st_cnt,
                               const int32_t* __restrict__ nnz, const int64_t* __restrict__ off, int64_t np,
                               int L, int64_t out_base, int32_t* __restrict__ col, int32_t* __restrict__ cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t p = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); p < np; p += warps) {
    const int m = nnz[p];
    const int64_t dst = out_base + off[p];
    for (int e = lane; e < m; e += 32) {
      col[dst + e] = st_col[p * L + e];
      cnt[dst + e] = st_cnt[p * L + e];
    }
  }
}

// One chunk's rows in the layout first_hit_counts hands back (view_factors.py:273-287): the
// origin patch id of every pair, its receiver and its count widened to int64, at the chunk's
// exclusive row offsets (one warp per row).
__global__ void k_compact_host(const int32_t* __restrict__ st_col, const int32_t* __restrict__ st_cnt,
                               const int32_t* __restrict__ nnz, const int64_t* __restrict__ off, int64_t np,
                               int L, int64_t first_id, int32_t* __restrict__ origin, int32_t* __restrict__ col,
                               int64_t* __restrict__ cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t p = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); p < np; p += warps) {
    const int m = nnz[p];
    const int64_t dst = off[p];
    for (int e = lane; e < m; e += 32) {
      origin[dst + e] = (int32_t)(first_id + p);
      col[dst + e] = st_col[p * L + e];
      cnt[dst + e] = st_cnt[p * L + e];
    }
  }
}

__global__ void k_i32_to_i64(const int32_t* __restrict__ in, int64_t* __restrict__ out, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    out[t] = in[t];
}

__global__ void k_fill_i64(int64_t* __restrict__ out, int64_t n, int64_t v) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    out[t] = v;
}

// ---------------------------------------------------------------------------- host

static void host_u128_mul(const pr_u128& a, const pr_u128& b, pr_u128& r) {
  unsigned __int128 x = ((unsigned __int128)a.hi << 64) | a.lo;
  unsigned __int128 y = ((unsigned __int128)b.hi << 64) | b.lo;
  unsigned __int128 z = x * y;
  r.lo = (uint64_t)z;
  r.hi = (uint64_t)(z >> 64);
}
static pr_u128 host_u128_add(const pr_u128& a, const pr_u128& b) {
  unsigned __int128 x = ((unsigned __int128)a.hi << 64) | a.lo;
  unsigned __int128 y = ((unsigned __int128)b.hi << 64) | b.lo;
  unsigned __int128 z = x + y;
  return pr_u128{(uint64_t)z, (uint64_t)(z >> 64)};
}

static pr_u128 host_affine(const pr_u128& A, const pr_u128& C, const pr_u128& x) {
  pr_u128 m;
  host_u128_mul(A, x, m);
  return host_u128_add(m, C);
}

// Seed tables on the device: kMapStride maps per seed, states (S), increments (S).
struct SeedTables {
  DevBuf<pr_u128> maps, state, inc;
  int build(const pr_pcg64* seeds, int S, cudaStream_t s) {
    std::vector<pr_u128> h_maps((size_t)S * kMapStride), h_state(S), h_inc(S);
    for (int q = 0; q < S; ++q) {
      pr_pcg64 sd;
      memcpy(&sd, seeds + q, sizeof(sd));  // seeds may be host memory only
      h_state[q] = pr_u128{sd.state_lo, sd.state_hi};
      h_inc[q] = pr_u128{sd.inc_lo, sd.inc_hi};
      pr_u128* m = h_maps.data() + (size_t)q * kMapStride;
      const pr_u128 A1{PR_PCG_MULT_LO, PR_PCG_MULT_HI}, C1 = h_inc[q];
      pr_u128 A = A1, C = C1;
      for (int i = 0; i < 64; ++i) {
        m[2 * i] = A;
        m[2 * i + 1] = C;
        // (A, C) o (A, C) = (A A, A C + C)
        pr_u128 AA, AC;
        host_u128_mul(A, A, AA);
        host_u128_mul(A, C, AC);
        C = host_u128_add(AC, C);
        A = AA;
      }
      // maps of n = 4 l steps by repeated composition with the one-step map
      pr_u128 An{1, 0}, Cn{0, 0};
      for (int n = 0; n <= 128; ++n) {
        if (n % 4 == 0 && n / 4 < 32) {
          m[kMapSmall + 2 * (n / 4)] = An;
          m[kMapSmall + 2 * (n / 4) + 1] = Cn;
        }
        if (n == 128) {
          m[kMapBatch] = An;
          m[kMapBatch + 1] = Cn;
        }
        // (A1, C1) o (An, Cn) = (A1 An, A1 Cn + C1)
        pr_u128 t;
        host_u128_mul(A1, An, t);
        Cn = host_affine(A1, C1, Cn);
        An = t;
      }
    }
    PR_TRY(maps.alloc(h_maps.size(), s));
    PR_TRY(state.alloc(S, s));
    PR_TRY(inc.alloc(S, s));
    PR_CUDA(cudaMemcpyAsync(maps.ptr, h_maps.data(), h_maps.size() * sizeof(pr_u128), cudaMemcpyHostToDevice, s));
    PR_CUDA(cudaMemcpyAsync(state.ptr, h_state.data(), S * sizeof(pr_u128), cudaMemcpyHostToDevice, s));
    PR_CUDA(cudaMemcpyAsync(inc.ptr, h_inc.data(), S * sizeof(pr_u128), cudaMemcpyHostToDevice, s));
    // the host vectors die at return: make the copies complete first
    PR_CUDA(cudaStreamSynchronize(s));
    return PR_OK;
  }
};

static Geom geom_of(const pr_case* c) {
  Geom g;
  g.occ = c->occ.ptr;
  g.ftab = c->ftab.ptr;
  g.nx = (int32_t)c->nx;
  g.ny = (int32_t)c->ny;
  g.nz = (int32_t)c->nz;
  g.n_cells = c->n_cells;
  return g;
}

static RaySrc src_of(const pr_case* c, const SeedTables& t) {
  RaySrc r;
  r.origin = c->origin.ptr;
  r.code = c->code.ptr;
  r.maps = t.maps.ptr;
  r.state = t.state.ptr;
  r.inc = t.inc.ptr;
  r.ny_d = (double)c->ny;
  r.nz_d = (double)c->nz;
  return r;
}

static int trace_grid() { return sm_count() * 8; }

// Variants of the pooled traversal: minimum resident blocks per SM (the register budget),
// cells per round (lookN: N occupancy loads in flight per lane) and rounds between lane refills.
// Every variant writes the same receivers; 6 blocks of 128 threads (80 registers, no spills) with
// two rounds of 8 cells were the fastest on 128^3 foam and layers and 96^3 fibers (7 blocks spill,
// and their pools leave the occupancy bits too little L1: 12 % slower; 4 blocks 20 %); shorter
// rounds win on small boxes.  The autotuner below picks the fastest per problem class by timing them
// on the first wave of the first call.
using TraceKernel = void (*)(const WaveChunk*, int, int, int, uint32_t*, int32_t*, unsigned long long*,
                             unsigned long long*);
struct TraceVariant {
  TraceKernel kernel;
  const char* name;
};
static const TraceVariant kVariants[] = {
    {k_trace_pool<6, 2, 8, false>, "6blk-look8x2"},
    {k_trace_pool<5, 2, 8, false>, "5blk-look8x2"},
    {k_trace_pool<6, 2, 6, false>, "6blk-look6x2"},
    {k_trace_pool<6, 4, 4, false>, "6blk-look4x4"},
};
static constexpr int kNumVariants = (int)(sizeof(kVariants) / sizeof(kVariants[0]));

static const TraceKernel kFlatKernel = k_trace_pool<6, 4, 2, true>;

// Largest unit of rays a warp takes at once (units shrink towards the end of a launch).
static constexpr int kMaxUnit = 2048;

// Persistent grid of a variant (kNumVariants: the walk of boxes without padded occupancy): as many blocks
// as fit on every SM.
static int variant_grid(int v) {
  static int blocks[kNumVariants + 1] = {0};
  if (blocks[v] == 0) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, v < kNumVariants ? kVariants[v].kernel : kFlatKernel, kWarps * 32,
                                                  0);
    blocks[v] = sm_count() * (per_sm > 0 ? per_sm : 1);
  }
  return blocks[v];
}

struct TuneKey {
  int64_t nx, ny, nz, L, cases;
  bool operator<(const TuneKey& o) const {
    return std::tie(nx, ny, nz, L, cases) < std::tie(o.nx, o.ny, o.nz, o.L, o.cases);
  }
};
static std::mutex g_tune_mu;
static std::map<TuneKey, int> g_tuned;
static int g_forced_variant = -1;
static int g_last_variant = 0;

}  // namespace pr

extern "C" {
// Force one traversal variant (0 .. count - 1), or -1 for the autotuner (default).
PR_API int pr_trace_set_variant(int v) {
  if (v < -1 || v >= pr::kNumVariants) {
    pr::set_error("traversal variant %d outside [-1, %d)", v, pr::kNumVariants);
    return PR_ERR_ARG;
  }
  std::lock_guard<std::mutex> lk(pr::g_tune_mu);
  pr::g_forced_variant = v;
  return PR_OK;
}
// Number of variants, the variant used by the last count pass, and its name (may be NULL).
PR_API int pr_trace_variant_info(int* count, int* last, const char** name) {
  std::lock_guard<std::mutex> lk(pr::g_tune_mu);
  if (count) *count = pr::kNumVariants;
  if (last) *last = pr::g_last_variant;
  if (name) *name = pr::kVariants[pr::g_last_variant].name;
  return PR_OK;
}
}

namespace pr {

struct WaveLaunch {
  const WaveChunk* chunks;  // device table
  int n_chunks;
  int total;                // global ray indices [0, total)
  bool padded;              // every chunk's case has its padded occupancy, or none has
  uint32_t* recv;           // hit codes, by global ray index
  int32_t* alone;           // scratch for the ray indices of k_trace_alone, one per ray
  unsigned long long* work; // work-unit counter, number of rays walked alone
  unsigned long long* ctr;  // 2 per chunk: DDA steps, failed rays
};

static int launch_variant(int v, const WaveLaunch& w, cudaStream_t s) {
  if (!w.padded) v = kNumVariants;
  PR_CUDA(cudaMemsetAsync(w.work, 0, 2 * sizeof(unsigned long long), s));
  const TraceKernel kernel = v < kNumVariants ? kVariants[v].kernel : kFlatKernel;
  ::pr::launch_mark(), kernel<<<variant_grid(v), kWarps * 32, 0, s>>>(
      w.chunks, w.n_chunks, w.total, kMaxUnit, w.recv, w.alone, w.work, w.ctr);
  PR_CUDA(cudaGetLastError());
  ::pr::launch_mark(), k_trace_alone<<<sm_count(), 128, 0, s>>>(w.chunks, w.n_chunks, w.recv, w.alone, w.work, w.ctr);
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}

// Variant for this problem class: forced, cached, or measured now on the given wave (each
// variant traces it once, timed with events; the per-chunk counters are cleared after).
static int choose_variant(const TuneKey& key, const WaveLaunch& w, cudaStream_t s, int* out) {
  *out = 0;
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    if (g_forced_variant >= 0) {
      *out = g_forced_variant;
      return PR_OK;
    }
    auto it = g_tuned.find(key);
    if (it != g_tuned.end()) {
      *out = it->second;
      return PR_OK;
    }
  }
  cudaEvent_t e0, e1;
  PR_CUDA(cudaEventCreate(&e0));
  PR_CUDA(cudaEventCreate(&e1));
  float best = 1e30f;
  int best_v = 0;
  for (int v = 0; v < kNumVariants; ++v) {
    PR_CUDA(cudaEventRecord(e0, s));
    PR_TRY(launch_variant(v, w, s));
    PR_CUDA(cudaEventRecord(e1, s));
    PR_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    PR_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (ms < best) {
      best = ms;
      best_v = v;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  PR_CUDA(cudaMemsetAsync(w.ctr, 0, 2 * sizeof(unsigned long long) * w.n_chunks, s));
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tuned[key] = best_v;
  }
  *out = best_v;
  return PR_OK;
}

int generate_rays(const pr_case* c, int64_t p0, int64_t p1, int64_t R, const pr_pcg64* seed, double* origins,
                  double* dirs, cudaStream_t s) {
  PR_ARG(p0 >= 0 && p1 >= p0 && p1 <= c->n_patches, "patch range [%lld, %lld) outside [0, %lld)",
         (long long)p0, (long long)p1, (long long)c->n_patches);
  PR_ARG(R >= 0, "rays_per_patch must be non-negative");
  const int64_t n = (p1 - p0) * R;
  if (n == 0) return PR_OK;
  SeedTables t;
  PR_TRY(t.build(seed, 1, s));
  DevBuf<double> o, d;
  PR_TRY(o.alloc(3 * n, s));
  PR_TRY(d.alloc(3 * n, s));
  ::pr::launch_mark(), k_generate<<<grid_for(n, 256, trace_grid()), 256, 0, s>>>(src_of(c, t), p0, p1 - p0, R, o.ptr, d.ptr);
  PR_CUDA(cudaGetLastError());
  PR_CUDA(cudaMemcpyAsync(origins, o.ptr, o.bytes(), cudaMemcpyDefault, s));
  PR_CUDA(cudaMemcpyAsync(dirs, d.ptr, d.bytes(), cudaMemcpyDefault, s));
  PR_CUDA(cudaStreamSynchronize(s));
  return PR_OK;
}

int trace_given(const pr_case* c, const double* origins, const double* dirs, int64_t n, int32_t* receiver,
                int64_t* n_failed, cudaStream_t s) {
  if (n_failed) *n_failed = 0;
  if (n == 0) return PR_OK;
  DevBuf<double> o, d;
  DevBuf<int32_t> rv;
  DevBuf<unsigned long long> ctr;
  PR_TRY(o.alloc(3 * n, s));
  PR_TRY(d.alloc(3 * n, s));
  PR_TRY(rv.alloc(n, s));
  PR_TRY(ctr.alloc(2, s));
  PR_CUDA(cudaMemcpyAsync(o.ptr, origins, o.bytes(), cudaMemcpyDefault, s));
  PR_CUDA(cudaMemcpyAsync(d.ptr, dirs, d.bytes(), cudaMemcpyDefault, s));
  PR_CUDA(cudaMemsetAsync(ctr.ptr, 0, ctr.bytes(), s));
  ::pr::launch_mark(), k_trace_given<<<grid_for(n, 256, trace_grid()), 256, 0, s>>>(geom_of(c), o.ptr, d.ptr, n, rv.ptr, ctr.ptr);
  PR_CUDA(cudaGetLastError());
  unsigned long long h[2];
  PR_CUDA(cudaMemcpyAsync(receiver, rv.ptr, rv.bytes(), cudaMemcpyDefault, s));
  PR_CUDA(cudaMemcpyAsync(h, ctr.ptr, sizeof(h), cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  if (n_failed) *n_failed = (int64_t)h[1];
  if (h[1]) {
    set_error("%lld rays did not resolve a receiving patch", (long long)h[1]);
    return PR_ERR_UNRESOLVED;
  }
  return PR_OK;
}

// Largest rays-per-origin segment the shared-memory sort handles (128 KiB of keys + heads).
static const int kMaxSegment = 16384;

// The per-patch sort's dynamic shared-memory limit is a per-device function attribute shared
// by every host thread: raise it once per device to the largest segment and never lower it.
static int enable_rle_smem() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  PR_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev >= 0 && dev < 64 && done[dev]) return PR_OK;
  PR_CUDA(cudaFuncSetAttribute(k_patch_rle, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(2 * kMaxSegment * sizeof(int32_t))));
  if (dev >= 0 && dev < 64) done[dev] = true;
  return PR_OK;
}

// Rays of one launch (a wave): chunks of one or more cases are packed until this bound.
static const int64_t kWaveRays = (int64_t)1 << 27;
// Rays per chunk.  A host pass takes smaller ones: its copies (16 bytes per pair) are as long as the
// tracing, so the first chunk's tracing and the last one's copy, which nothing overlaps, have to be
// short (128^3 foam, 2.6e8 rays: 56.7 ms with chunks of 2^26 rays, 50.9 with 2^24; 151 x 77 x 93
// layers, 6e7 rays: 16.0 and 13.7 ms).  Chunks of 2^22 rays cost more in launches and round trips
// than they save (16.0 ms).
static const int64_t kChunkRays = (int64_t)1 << 26, kHostChunkRays = (int64_t)1 << 24;

// Per-case accumulation of a batched count pass.
struct CaseCounts {
  std::unique_ptr<pr_counts> k;
  DevBuf<int64_t> nnz_all;  // row lengths
  struct Piece {
    DevBuf<int32_t> col, cnt;
    int64_t n = 0;
  };
  std::vector<Piece> pieces;  // compacted chunks in patch order
};

// A count pass of one case that hands its edge list to host memory while it runs: each
// chunk's rows, once compacted, are laid out as first_hit_counts returns them and copied on a
// stream of their own into origin / receiver / count at their place in the sorted list, while
// the next chunks trace; no device table is kept.
struct HostSink {
  int32_t* origin;
  int32_t* receiver;
  int64_t* count;
  int64_t capacity;  // pairs the arrays hold
  int64_t written = 0;
};

namespace {
// The copy stream of a host pass and what its copies read, released in this order: the stream
// is drained before the device buffers go back to the cache.
struct HostPass {
  struct Piece {
    DevBuf<int32_t> o, r;
    DevBuf<int64_t> c;
  };
  std::vector<Piece> pieces;
  std::vector<cudaEvent_t> events;
  cudaStream_t copy = nullptr;
  ~HostPass() {
    if (copy) {
      cudaStreamSynchronize(copy);
      cudaStreamDestroy(copy);
    }
    for (cudaEvent_t e : events) cudaEventDestroy(e);
    pieces.clear();
  }
};
}  // namespace

// first_hit_counts for n_cases geometries at once (view_factors.py:273-300 per case): every
// case traces rays_per_patch rays per patch for each of its S seeds (seeds[c * S + s]);
// chunks of all cases share persistent launches of the pooled traversal.  With `sink` (one
// case), the edge list goes to host memory as the chunks finish and `out` is not used.
int counts_batch(const pr_case* const* cases, int nc, int64_t R, const pr_pcg64* seeds, int S, cudaStream_t s,
                 pr_counts** out, HostSink* sink) {
  PR_ARG(nc > 0, "no cases");
  PR_ARG(!sink || nc == 1, "a host pass takes one case");
  PR_ARG(R > 0 && S > 0, "rays_per_patch and the number of seeds must be positive");
  const int64_t L64 = R * S;
  if (L64 > kMaxSegment) {
    set_error("%lld rays per origin patch exceed the %d supported in one call", (long long)L64, kMaxSegment);
    return PR_ERR_LIMIT;
  }
  const int L = (int)L64;
  int Lpad = 1;
  while (Lpad < L) Lpad <<= 1;
  if (Lpad < 64) Lpad = 64;
  int dev0 = 0;
  cudaGetDevice(&dev0);

  // seed tables and per-case outputs
  std::vector<SeedTables> tables(nc);
  std::vector<CaseCounts> cc(nc);
  for (int c = 0; c < nc; ++c) {
    PR_ARG(cases[c] != nullptr, "case %d is NULL", c);
    PR_ARG(cases[c]->device == dev0, "case %d lives on another device", c);
    // int32 hit codes (and cell indices)
    if (6 * cases[c]->n_cells + 2 * cases[c]->ny * cases[c]->nz > (int64_t)INT32_MAX) {
      set_error("case %d: %lld cells exceed the int32 hit codes of the traversal", c, (long long)cases[c]->n_cells);
      return PR_ERR_LIMIT;
    }
    PR_TRY(tables[c].build(seeds + (size_t)c * S, S, s));
    const int64_t P = cases[c]->n_patches;
    cc[c].k.reset(new pr_counts());
    cc[c].k->device = dev0;
    cc[c].k->csr = std::make_shared<CountCsr>();
    cc[c].k->csr->n_rows = P;
    PR_TRY(cc[c].k->csr->row_ptr.alloc(P + 1, s));
    PR_TRY(cc[c].k->rays.alloc(P > 0 ? P : 1, s));
    PR_TRY(cc[c].nnz_all.alloc(P > 0 ? P : 1, s));
    if (P > 0) {
      ::pr::launch_mark(), k_fill_i64<<<grid_for(P, 256), 256, 0, s>>>(cc[c].k->rays.ptr, P, L64);
      PR_CUDA(cudaGetLastError());
    }
  }

  // chunks: (case, first patch, patches), those of cases with padded occupancy first
  struct Chunk {
    int c;
    int64_t p0, np;
  };
  std::vector<Chunk> chunks;
  const int64_t chunk_patches = std::max<int64_t>(1, (sink ? kHostChunkRays : kChunkRays) / L64);
  for (bool pad : {true, false})
    for (int c = 0; c < nc; ++c)
      for (int64_t p0 = 0; (cases[c]->pad.ptr != nullptr) == pad && p0 < cases[c]->n_patches; p0 += chunk_patches)
        chunks.push_back({c, p0, std::min(chunk_patches, cases[c]->n_patches - p0)});

  // wave buffers
  int64_t wave_cap = 0;
  for (const Chunk& ch : chunks) wave_cap = std::max(wave_cap, ch.np * L64);
  wave_cap = std::max(wave_cap, std::min<int64_t>(kWaveRays, [&] {
                        int64_t t = 0;
                        for (const Chunk& ch : chunks) t += ch.np * L64;
                        return t;
                      }()));
  if (sink) {
    // one chunk per wave, so that every chunk's copy overlaps the next chunk's traversal
    wave_cap = 0;
    for (const Chunk& ch : chunks) wave_cap = std::max(wave_cap, ch.np * L64);
  }
  HostPass hp;
  if (sink) PR_CUDA(cudaStreamCreateWithFlags(&hp.copy, cudaStreamNonBlocking));
  DevBuf<uint32_t> recv;
  DevBuf<int32_t> st_col, st_cnt, nnz;
  DevBuf<int64_t> off;
  DevBuf<unsigned long long> work, ctr;
  DevBuf<WaveChunk> dchunks;
  DevBuf<RleChunk> drle;
  const int64_t max_wave_patches = wave_cap / L64 + (int64_t)chunks.size();
  // hit codes by wave-wide ray index: chunk starts are multiples of kAlign
  PR_TRY(recv.alloc(wave_cap + (int64_t)chunks.size() * kAlign, s));
  PR_TRY(st_col.alloc(wave_cap, s));
  PR_TRY(st_cnt.alloc(wave_cap, s));
  PR_TRY(nnz.alloc(max_wave_patches, s));
  PR_TRY(off.alloc(max_wave_patches + 1, s));
  PR_TRY(work.alloc(2, s));
  PR_TRY(ctr.alloc(2 * chunks.size(), s));
  PR_TRY(dchunks.alloc(chunks.size(), s));
  PR_TRY(drle.alloc(chunks.size(), s));
  PR_CUDA(cudaMemsetAsync(ctr.ptr, 0, ctr.bytes(), s));
  PR_TRY(enable_rle_smem());
  const size_t smem = (size_t)2 * Lpad * sizeof(int32_t);
  const int rle_threads = Lpad >= 1024 ? 512 : (Lpad >= 256 ? 256 : 64);
  size_t scan_bytes = 0;
  PR_CUDA(cub::DeviceScan::InclusiveSum(nullptr, scan_bytes, off.ptr, off.ptr + 1, max_wave_patches, s));
  DevBuf<uint8_t> scan_tmp;
  PR_TRY(scan_tmp.alloc(scan_bytes + 16, s));

  int variant = 0;
  bool tuned = false;
  std::vector<WaveChunk> hw;
  std::vector<RleChunk> hr;
  std::vector<int64_t> totals;
  for (size_t w0 = 0; w0 < chunks.size();) {
    // pack a wave, of cases that are walked alike
    const bool padded = cases[chunks[w0].c]->pad.ptr != nullptr;
    size_t w1 = w0;
    int64_t rays = 0;
    while (w1 < chunks.size() && (cases[chunks[w1].c]->pad.ptr != nullptr) == padded &&
           (w1 == w0 || rays + chunks[w1].np * L64 <= wave_cap))
      rays += chunks[w1++].np * L64;
    const int nw = (int)(w1 - w0);
    hw.assign(nw, WaveChunk{});
    hr.assign(nw, RleChunk{});
    int64_t start = 0, ray0 = 0, patch0 = 0;
    for (int k = 0; k < nw; ++k) {
      const Chunk& ch = chunks[w0 + k];
      const pr_case* c = cases[ch.c];
      WaveChunk& W = hw[k];
      W.occ = c->occ.ptr;
      W.pad = c->pad.ptr;
      W.box = c->box;
      W.origin = c->origin.ptr;
      W.code = c->code.ptr;
      W.maps = tables[ch.c].maps.ptr;
      W.state = tables[ch.c].state.ptr;
      W.inc = tables[ch.c].inc.ptr;
      W.n = ch.np * L64;
      W.np = ch.np;
      W.p0 = ch.p0;
      W.R = R;
      W.start = start;
      W.n_cells = c->n_cells;
      W.ny_d = (double)c->ny;
      W.nz_d = (double)c->nz;
      hr[k] = RleChunk{recv.ptr + start, c->ftab.ptr, c->box, ctr.ptr + 2 * (w0 + k) + 1, ch.np, patch0, ray0};
      start += (W.n + kAlign - 1) / kAlign * kAlign;
      ray0 += W.n;
      patch0 += ch.np;
    }
    const int64_t total = hw[nw - 1].start + hw[nw - 1].n;
    PR_CUDA(cudaMemcpyAsync(dchunks.ptr, hw.data(), nw * sizeof(WaveChunk), cudaMemcpyHostToDevice, s));
    PR_CUDA(cudaMemcpyAsync(drle.ptr, hr.data(), nw * sizeof(RleChunk), cudaMemcpyHostToDevice, s));
    unsigned long long* wave_ctr = ctr.ptr + 2 * w0;
    WaveLaunch wl{dchunks.ptr, nw, (int)total, padded, recv.ptr, st_col.ptr, work.ptr, wave_ctr};
    if (padded && !tuned) {
      const pr_case* c0 = cases[chunks[w0].c];
      PR_TRY(choose_variant(TuneKey{c0->nx, c0->ny, c0->nz, L64, nc}, wl, s, &variant));
      tuned = true;
    }
    ::pr::timer_begin(kTimerTrace, s);
    PR_TRY(launch_variant(variant, wl, s));
    ::pr::timer_end(kTimerTrace, s);
    const int rle_grid = (int)std::min<int64_t>(patch0, (int64_t)sm_count() * 16);
    ::pr::timer_begin(kTimerRle, s);
    if (Lpad <= 1024) {
      const int wg = (int)std::min<int64_t>((patch0 + 3) / 4, (int64_t)sm_count() * 32);
      auto kern = Lpad <= 64 ? k_patch_rle_warp<2> : Lpad <= 128 ? k_patch_rle_warp<4>
                : Lpad <= 256 ? k_patch_rle_warp<8> : Lpad <= 512 ? k_patch_rle_warp<16> : k_patch_rle_warp<32>;
      ::pr::launch_mark(), kern<<<wg, 128, 0, s>>>(drle.ptr, nw, patch0, L, (int)R, st_col.ptr, st_cnt.ptr, nnz.ptr);
    } else
    ::pr::launch_mark(), k_patch_rle<<<rle_grid, rle_threads, smem, s>>>(drle.ptr, nw, patch0, L, (int)R, Lpad,
                                                                     st_col.ptr, st_cnt.ptr, nnz.ptr);
    ::pr::timer_end(kTimerRle, s);
    PR_CUDA(cudaGetLastError());
    // per chunk: row lengths into the case, exclusive offsets for the compaction
    totals.assign(nw, 0);
    for (int k = 0; k < nw; ++k) {
      const Chunk& ch = chunks[w0 + k];
      const RleChunk& rc = hr[k];
      ::pr::launch_mark(), k_i32_to_i64<<<grid_for(ch.np, 256), 256, 0, s>>>(nnz.ptr + rc.patch0,
                                                                            cc[ch.c].nnz_all.ptr + ch.p0, ch.np);
      PR_CUDA(cudaGetLastError());
      int64_t* o = off.ptr + rc.patch0 + k;  // np + 1 slots per chunk
      PR_CUDA(cudaMemsetAsync(o, 0, sizeof(int64_t), s));
      PR_CUDA(cub::DeviceScan::InclusiveSum(scan_tmp.ptr, scan_bytes, cc[ch.c].nnz_all.ptr + ch.p0, o + 1, ch.np, s));
      PR_CUDA(cudaMemcpyAsync(&totals[k], o + ch.np, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    }
    PR_CUDA(cudaStreamSynchronize(s));
    for (int k = 0; k < nw && sink; ++k) {
      const Chunk& ch = chunks[w0 + k];
      const RleChunk& rc = hr[k];
      const int64_t n = totals[k];
      if (sink->written + n > sink->capacity) {
        set_error("the edge list exceeds the %lld pairs the host arrays hold", (long long)sink->capacity);
        return PR_ERR_LIMIT;
      }
      HostPass::Piece pc;
      PR_TRY(pc.o.alloc(n > 0 ? n : 1, s));
      PR_TRY(pc.r.alloc(n > 0 ? n : 1, s));
      PR_TRY(pc.c.alloc(n > 0 ? n : 1, s));
      ::pr::launch_mark(), k_compact_host<<<grid_for(ch.np * 32, 256), 256, 0, s>>>(
          st_col.ptr + rc.ray0, st_cnt.ptr + rc.ray0, nnz.ptr + rc.patch0, off.ptr + rc.patch0 + k, ch.np, L, ch.p0,
          pc.o.ptr, pc.r.ptr, pc.c.ptr);
      PR_CUDA(cudaGetLastError());
      cudaEvent_t ev = nullptr;
      PR_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
      hp.events.push_back(ev);
      PR_CUDA(cudaEventRecord(ev, s));
      PR_CUDA(cudaStreamWaitEvent(hp.copy, ev, 0));
      if (n > 0) {
        const int64_t at = sink->written;
        PR_CUDA(cudaMemcpyAsync(sink->origin + at, pc.o.ptr, (size_t)n * 4, cudaMemcpyDeviceToHost, hp.copy));
        PR_CUDA(cudaMemcpyAsync(sink->receiver + at, pc.r.ptr, (size_t)n * 4, cudaMemcpyDeviceToHost, hp.copy));
        PR_CUDA(cudaMemcpyAsync(sink->count + at, pc.c.ptr, (size_t)n * 8, cudaMemcpyDeviceToHost, hp.copy));
      }
      sink->written += n;
      hp.pieces.push_back(std::move(pc));
    }
    for (int k = 0; k < nw && !sink; ++k) {
      const Chunk& ch = chunks[w0 + k];
      const RleChunk& rc = hr[k];
      CaseCounts::Piece pc;
      pc.n = totals[k];
      PR_TRY(pc.col.alloc(pc.n > 0 ? pc.n : 1, s));
      PR_TRY(pc.cnt.alloc(pc.n > 0 ? pc.n : 1, s));
      ::pr::launch_mark(), k_compact_rows<<<grid_for(ch.np * 32, 256), 256, 0, s>>>(
          st_col.ptr + rc.ray0, st_cnt.ptr + rc.ray0, nnz.ptr + rc.patch0, off.ptr + rc.patch0 + k, ch.np, L, 0,
          pc.col.ptr, pc.cnt.ptr);
      PR_CUDA(cudaGetLastError());
      cc[ch.c].pieces.push_back(std::move(pc));
    }
    // the next wave's kernels reuse the stage buffers after these compactions in stream order
    w0 = w1;
  }

  // per case: concatenate the pieces, row offsets, counters
  std::vector<unsigned long long> hctr(2 * chunks.size());
  PR_CUDA(cudaMemcpyAsync(hctr.data(), ctr.ptr, ctr.bytes(), cudaMemcpyDeviceToHost, s));
  PR_CUDA(cudaStreamSynchronize(s));
  int64_t failed = 0;
  std::vector<int64_t> steps(nc, 0), fails(nc, 0);
  for (size_t k = 0; k < chunks.size(); ++k) {
    steps[chunks[k].c] += (int64_t)hctr[2 * k];
    fails[chunks[k].c] += (int64_t)hctr[2 * k + 1];
  }
  if (sink) {
    PR_CUDA(cudaStreamSynchronize(hp.copy));
    {
      std::lock_guard<std::mutex> lk(g_tune_mu);
      g_last_variant = variant;
    }
    if (fails[0]) {
      set_error("%lld rays did not resolve a receiving patch", (long long)fails[0]);
      return PR_ERR_UNRESOLVED;
    }
    return PR_OK;
  }
  for (int c = 0; c < nc; ++c) {
    CountCsr& csr = *cc[c].k->csr;
    const int64_t P = csr.n_rows;
    int64_t total = 0;
    for (auto& pc : cc[c].pieces) total += pc.n;
    csr.nnz = total;
    PR_TRY(csr.col.alloc(total > 0 ? total : 1, s));
    PR_TRY(csr.cnt.alloc(total > 0 ? total : 1, s));
    int64_t at = 0;
    for (auto& pc : cc[c].pieces) {
      if (pc.n) {
        PR_CUDA(cudaMemcpyAsync(csr.col.ptr + at, pc.col.ptr, pc.n * 4, cudaMemcpyDeviceToDevice, s));
        PR_CUDA(cudaMemcpyAsync(csr.cnt.ptr + at, pc.cnt.ptr, pc.n * 4, cudaMemcpyDeviceToDevice, s));
      }
      at += pc.n;
    }
    cc[c].pieces.clear();
    PR_CUDA(cudaMemsetAsync(csr.row_ptr.ptr, 0, sizeof(int64_t), s));
    if (P > 0) {
      size_t b = 0;
      PR_CUDA(cub::DeviceScan::InclusiveSum(nullptr, b, cc[c].nnz_all.ptr, csr.row_ptr.ptr + 1, P, s));
      DevBuf<uint8_t> tmp;
      PR_TRY(tmp.alloc(b + 16, s));
      PR_CUDA(cub::DeviceScan::InclusiveSum(tmp.ptr, b, cc[c].nnz_all.ptr, csr.row_ptr.ptr + 1, P, s));
    }
    cc[c].k->rays_traced = P * L64;
    cc[c].k->dda_steps = steps[c];
    cc[c].k->last_stream = s;
    failed += fails[c];
  }
  PR_CUDA(cudaStreamSynchronize(s));
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_last_variant = variant;
  }
  if (failed) {
    set_error("%lld rays did not resolve a receiving patch", (long long)failed);
    return PR_ERR_UNRESOLVED;
  }
  for (int c = 0; c < nc; ++c) out[c] = cc[c].k.release();
  return PR_OK;
}

int first_hit_counts(const pr_case* c, int64_t R, const pr_pcg64* seeds, int S, cudaStream_t s, pr_counts** out) {
  return counts_batch(&c, 1, R, seeds, S, s, out, nullptr);
}

int first_hit_counts_host(const pr_case* c, int64_t R, const pr_pcg64* seeds, int S, cudaStream_t s,
                          int32_t* origin, int32_t* receiver, int64_t* count, int64_t capacity, int64_t* n_pairs) {
  HostSink sink{origin, receiver, count, capacity, 0};
  *n_pairs = 0;
  PR_TRY(counts_batch(&c, 1, R, seeds, S, s, nullptr, &sink));
  *n_pairs = sink.written;
  return PR_OK;
}

}  // namespace pr
