// 2D levels of the V-cycle by tiles (sm_103a): two whole red-black sweeps of a
// level, with the restriction behind them or the prolongation before them, in one
// launch.
//
// A level that fits in L2 is bound by the latency of its launches: ten of them,
// each 1.5 to 2.5 us even when the next one's start overlaps, for nanoseconds of
// work.  Here a block loads its tile with a halo as deep as the colours it will
// relax (one cell more in front of a restriction), relaxes the colours one after
// the other in shared memory on a region that shrinks by a cell each time, and
// stores the tile: the halo is relaxed again by the neighbours instead of being
// exchanged, so a level is two launches.  Neighbouring blocks still read the
// tile's old values, so the unknown alternates between two arrays.  Each cell's
// arithmetic and its order are those of the separate launches (mg_cells.cuh,
// kernels_split.cu): the iterates keep their bits.
//
// Every array in shared memory has the halo's cells outside the grid as zeros; a
// wall's coefficient is a zero, so a stencil has no bounds tests.  The
// coefficients, which no kernel of the cycle writes, are loaded (on the
// colour-split level formed from the density, once for all colours) before the
// wait for the preceding kernel: ordinary launches separate the set-up that
// wrote them from the cycle.
//
// Time of a solve per cycle, separate launches -> tiles: FP64 128^2 75.1 -> 48.4 us,
// 512^2 166 -> 119; mixed 128 x 256 52.9 -> 35.4, 512^2 79.5 -> 50.5, 1024^2 (from level
// 512^2 down) 114.5 -> 89.5.  Tiles of 16 x 8 cells with 256 threads: more threads than
// cells of a colour, since a phase is one chain of latencies (FP64 128^2 a third slower
// with 128 threads, a fifth to a third with 16 x 16 and 32 x 16 tiles).  The split level
// takes 32 x 16 with 512 (16 x 8 is a tenth slower): its blocks also form their
// coefficients.
#include <algorithm>

#include "gbmg_internal.h"
#include "mg_cells.cuh"
#include "pdl.cuh"

namespace gbmg {

namespace {

// kM: colours relaxed; kRes: followed by the restriction; kSplit: the colour-split
// finest level, coefficients from the density; kHalf (FP64): restrict_cell's half
template <typename T, int kTx, int kTy, int kM, bool kRes, int kThr, bool kSplit = false,
          bool kHalf = false>
struct Tile {
  using Value = T;
  static constexpr int H = kM + (kRes ? 1 : 0);  // even in front of a prolongation
  static constexpr int TX = kTx, TY = kTy, M = kM, THREADS = kThr;
  static constexpr bool RES = kRes, SPLIT = kSplit, HALF = kHalf, IDIAG = sizeof(T) == 8;
  static constexpr int LX = kTx + 2 * H, LY = kTy + 2 * H, N = LX * LY;
  static constexpr size_t BYTES = (size_t)(IDIAG ? 5 : 4) * N * sizeof(T);
};

struct TileArgs {
  int first;     // colour relaxed first
  int zero;      // from a zero guess (sol_in is not read)
  int prolong;   // add the interpolated coarse unknown first
};

// sol_in -> sol_out
template <typename P>
__global__ void __launch_bounds__(P::THREADS)
    k_tile(LevelView<typename P::Value> F, LevelView<typename P::Value> C,
           const typename P::Value* __restrict__ sol_in, typename P::Value* __restrict__ sol_out,
           TileArgs A) {
  using T = typename P::Value;
  using V2 = typename cells::Vec2<T>::type;
  constexpr int H = P::H, LX = P::LX, LY = P::LY, N = P::N;
  pdl_launch();
  extern __shared__ __align__(16) unsigned char tile_raw[];
  T* const sol = reinterpret_cast<T*>(tile_raw);
  T* const src = sol + N;
  T* const cx = src + N;
  T* const cy = cx + N;
  T* const id = cy + N;  // FP64
  const int tid = threadIdx.x;
  const int nx = F.nx, ny = F.ny;
  const int bx = blockIdx.x * P::TX - H, by = blockIdx.y * P::TY - H;  // of local cell (0, 0)
  // a cell's place in the unknown, the right-hand side and the density
  const auto at = [&](int x, int y) {
    const size_t q = (size_t)y * nx + x;
    return P::SPLIT ? (size_t)((x + y) & 1) * F.hstride + (q >> 1) : q;
  };
  const auto inside = [&](int x, int y) {
    return (unsigned)x < (unsigned)nx && (unsigned)y < (unsigned)ny;
  };
#pragma unroll 4
  for (int t = tid; t < N; t += P::THREADS) {
    const int ly = t / LX, x = bx + t - ly * LX, y = by + ly;
    const bool in = inside(x, y);
    if constexpr (P::SPLIT) {
      sol[t] = in ? F.rho[at(x, y)] : T(0);  // (the density, for now)
    } else {
      const size_t q = in ? at(x, y) : 0;
      cx[t] = in ? F.cx[q] : T(0);
      cy[t] = in ? F.cy[q] : T(0);
      if (P::IDIAG) id[t] = in ? F.idiag[q] : T(0);
    }
  }
  if constexpr (P::SPLIT) {
    __syncthreads();
    // low faces; those of the region's first row and column are not read
    for (int t = tid; t < N; t += P::THREADS) {
      const int ly = t / LX, lx = t - ly * LX, x = bx + lx, y = by + ly;
      const bool in = inside(x, y);
      cx[t] = in && lx > 0 && x > 0 ? rho_face32(F.kx, sol[t], sol[t - 1]) : T(0);
      cy[t] = in && ly > 0 && y > 0 ? rho_face32(F.ky, sol[t], sol[t - LX]) : T(0);
    }
    __syncthreads();
  }
  pdl_wait();
#pragma unroll 4
  for (int t = tid; t < N; t += P::THREADS) {
    const int ly = t / LX, x = bx + t - ly * LX, y = by + ly;
    const bool in = inside(x, y);
    const size_t q = in ? at(x, y) : 0;
    src[t] = in ? __ldcg(F.src + q) : T(0);
    if (!A.prolong) sol[t] = in && !A.zero ? __ldcg(sol_in + q) : T(0);
  }
  if (!P::RES && A.prolong) {
    // sol_in + the coarse unknown's central-slope interpolation (prolong_cell);
    // both axes are halved, so the region is made of whole coarse cells
    constexpr int KX = LX / 2, KY = LY / 2;
    const T* e = C.sol;
    for (int t = tid; t < KX * KY; t += P::THREADS) {
      const int lj = t / KX, li = t - lj * KX;
      const int I = (bx >> 1) + li, J = (by >> 1) + lj;
      T* o = sol + 2 * lj * LX + 2 * li;
      if ((unsigned)I >= (unsigned)C.nx || (unsigned)J >= (unsigned)C.ny) {
        o[0] = o[1] = o[LX] = o[LX + 1] = T(0);
        continue;
      }
      const T* ep = e + (size_t)J * C.nx + I;
      const T ec = __ldcg(ep);
      const T xp = I < C.nx - 1 ? __ldcg(ep + 1) : ec, xm = I > 0 ? __ldcg(ep - 1) : ec;
      const T yp = J < C.ny - 1 ? __ldcg(ep + C.nx) : ec, ym = J > 0 ? __ldcg(ep - C.nx) : ec;
      const T mx = T(0.5) * (xp - xm), my = T(0.5) * (yp - ym);
#pragma unroll
      for (int dy = 0; dy < 2; ++dy) {
        V2 cur;
        if constexpr (P::SPLIT) {
          cur.x = __ldcg(sol_in + at(2 * I, 2 * J + dy));
          cur.y = __ldcg(sol_in + at(2 * I + 1, 2 * J + dy));
        } else {
          cur = __ldcg(reinterpret_cast<const V2*>(sol_in + at(2 * I, 2 * J + dy)));
        }
        const T ty = dy ? T(0.25) * my : -(T(0.25) * my);
        T v0 = ec + -(T(0.25) * mx), v1 = ec + T(0.25) * mx;
        v0 += ty;
        v1 += ty;
        o[dy * LX] = cur.x + v0;
        o[dy * LX + 1] = cur.y + v1;
      }
    }
  }
  __syncthreads();
  const auto neighbours = [&](int q, T& s, T& d) {
    T c;
    s = T(0);
    c = cx[q]; s += c * sol[q - 1]; d = c;
    c = cx[q + 1]; s += c * sol[q + 1]; d += c;
    c = cy[q]; s += c * sol[q - LX]; d += c;
    c = cy[q + LX]; s += c * sol[q + LX]; d += c;
  };
#pragma unroll
  for (int p = 1; p <= P::M; ++p) {
    // local cells p .. L - p - 1 of each axis
    const int W = (LX - 2 * p) / 2, NY = LY - 2 * p;
    const int colour = A.first ^ ((p - 1) & 1);
#pragma unroll 2
    for (int t = tid; t < W * NY; t += P::THREADS) {
      const int r = t / W, m = t - r * W, ly = p + r, y = by + ly;
      const int lx = p + 2 * m + ((colour + bx + p + y) & 1);
      if (!inside(bx + lx, y)) continue;
      const int q = ly * LX + lx;
      T s, d;
      neighbours(q, s, d);
      if (A.zero && p == 1) s = T(0);  // (the level's values are taken as zero)
      if constexpr (P::SPLIT) sol[q] = rho_relax32(s, src[q], d);
      else if constexpr (P::IDIAG) sol[q] = (s - src[q]) * id[q];
      else sol[q] = (s - src[q]) / d;
    }
    __syncthreads();
  }
  for (int t = tid; t < P::TX * P::TY; t += P::THREADS) {
    const int ty = t / P::TX, tx = t - ty * P::TX;
    const int x = bx + H + tx, y = by + H + ty;
    if (inside(x, y)) sol_out[at(x, y)] = sol[(ty + H) * LX + tx + H];
  }
  if (!P::RES) return;
  // residuals in place of the right-hand side, which only their own cells read
  // (HALF: the children of the colour relaxed last, 1, have none)
  constexpr int SX = P::HALF ? 2 : 1, RX = P::TX / SX;
  for (int t = tid; t < RX * P::TY; t += P::THREADS) {
    const int y = t / RX;
    int x = t - y * RX;
    if (P::HALF) x = 2 * x + (y & 1);
    const int q = (y + H) * LX + x + H;
    T s, d;
    neighbours(q, s, d);
    src[q] = src[q] - (s - d * sol[q]);
  }
  __syncthreads();
  // the mean over the children (y, x)
  constexpr int CX = P::TX / 2, CY = P::TY / 2;
  for (int t = tid; t < CX * CY; t += P::THREADS) {
    const int j = t / CX, i = t - j * CX;
    const int I = blockIdx.x * CX + i, J = blockIdx.y * CY + j;
    if (I >= C.nx || J >= C.ny) continue;
    const T* r = src + (2 * j + H) * LX + 2 * i + H;
    T acc = T(0);
#pragma unroll
    for (int dy = 0; dy < 2; ++dy)
#pragma unroll
      for (int dx = 0; dx < 2; ++dx)
        if (!P::HALF || dx == dy) acc += r[dy * LX + dx];
    C.src[(size_t)J * C.nx + I] = acc * T(0.25);
  }
}

template <typename P>
void tile_launch(cudaStream_t s, const LevelView<typename P::Value>& F,
                 const LevelView<typename P::Value>& C, const typename P::Value* in,
                 typename P::Value* out, const TileArgs& A) {
  const dim3 grd((unsigned)((F.nx + P::TX - 1) / P::TX), (unsigned)((F.ny + P::TY - 1) / P::TY));
  static_assert(P::BYTES <= 48 * 1024, "static limit");
  launch_pdl(k_tile<P>, grd, dim3(P::THREADS), P::BYTES, s, F, C, in, out, A);
}

template <typename T, bool R, bool kHalf>
void tile_pick(cudaStream_t s, const LevelView<T>& F, const LevelView<T>& C, const T* in, T* out,
               int sweeps, const TileArgs& A) {
  if constexpr (sizeof(T) == 4) {
    if (F.split) {
      if (sweeps == 2) tile_launch<Tile<T, 32, 16, 4, R, 512, true>>(s, F, C, in, out, A);
      else tile_launch<Tile<T, 32, 16, 2, R, 512, true>>(s, F, C, in, out, A);
      return;
    }
  }
  if (sweeps == 2) tile_launch<Tile<T, 16, 8, 4, R, 256, false, kHalf>>(s, F, C, in, out, A);
  else tile_launch<Tile<T, 16, 8, 2, R, 256, false, kHalf>>(s, F, C, in, out, A);
}

}  // namespace

// 2D levels of at most 512 x 512 cells, both axes halved (so that the halo is made
// of whole coarse cells and rows are even).  Larger levels are bound by their
// arithmetic and traffic, which the halos double.  Time of a solve per cycle with
// the finest level in separate launches -> in tiles (all below it in tiles): 1024^2 FP64 237 ->
// 272 us, colour-split FP32 89.5 -> 102.8, FP32 with stored coefficients 96.0 -> 96.0;
// 768^2 178.5 -> 187.1, 74.4 -> 73.5, 74.3 -> 74.1; below that tiles are ahead (768 x
// 512 177 -> 145, 70.4 -> 64.6, 68.3 -> 68.3), so the line is on the safe side.  3D
// halos cost more: 32^3 in tiles of 8^3 leaves the 256^3 cycle as it was (463.5 for
// 465.6 us), 64^3 in tiles of 16 x 8 x 8, a sweep a launch, makes it 474.
bool tile_level(int nx, int ny, int nz, int fx, int fy) {
  return nz == 1 && fx == 2 && fy == 2 && (size_t)nx * ny <= (size_t)1 << 18;
}

template <typename T>
void launch_tile(cudaStream_t s, const LevelView<T>& F, const LevelView<T>& C, const T* in, T* out,
                 int sweeps, int first, TileEnds e, bool half) {
  const TileArgs A{first, e == kTileZero || e == kTileZeroRestrict, e == kTileProlong};
  if (e == kTileRestrict || e == kTileZeroRestrict) {
    if constexpr (sizeof(T) == 8)
      if (half) return tile_pick<T, true, true>(s, F, C, in, out, sweeps, A);
    tile_pick<T, true, false>(s, F, C, in, out, sweeps, A);
  } else {
    tile_pick<T, false, false>(s, F, C, in, out, sweeps, A);
  }
}

template void launch_tile<float>(cudaStream_t, const LevelView<float>&, const LevelView<float>&,
                                 const float*, float*, int, int, TileEnds, bool);
template void launch_tile<double>(cudaStream_t, const LevelView<double>&, const LevelView<double>&,
                                  const double*, double*, int, int, TileEnds, bool);

}  // namespace gbmg
