// 2D TM (Ez, Hx, Hy) Yee kernels for sm_100a.
//
// One step of the reference's scan body (jaxphys src/neurosim/em/fdtd.py:304-357):
//   Hx[:, :-1] -= a (Ez[:, 1:] - Ez[:, :-1])                 (:325-327)
//   Hy[:-1, :] += a (Ez[1:, :] - Ez[:-1, :])                 (:330-332)
//   Ez[1:, 1:] += b ((Hy[i]-Hy[i-1]) - (Hx[j]-Hx[j-1]))       (:335-340)
//   periodic: the same with wrap-around differences on every cell (:314-321)
// then, by boundary mode: damping exp(-sigma_avg dt/eps0) (:342-344), mirrored
// edges (:264-282) or wrapped edges (:284-302); then line sources on whole
// rows Ez[:, y] (:257-262,354) and conductor rows forced to 0 (:357).
#pragma once

#include "fdtd_common.cuh"

namespace jxf {

struct Step2D {
  int nx, ny;
  float a, b;
  float* ez;
  float* hx;
  float* hy;
  const float* damp[2];  // separable damping (ABSORBING)
  // line sources (list order)
  int n_src;
  const int* src_y;
  const float* src_amp;
  const int* src_wave;
  const float* wave;
  long long wave_len;
  long long step;
  // conductor rows
  int n_wall;
  const int* wall_y;
  const int* wall_g0;  // < 0: solid
  const int* wall_g1;
};

template <int MODE>
__global__ void __launch_bounds__(256) k2d_h(const __grid_constant__ Step2D p) {
  const int nx = p.nx, ny = p.ny;
  const long long n = (long long)nx * ny;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(idx % ny);
    const int x = (int)(idx / ny);
    const float e = p.ez[idx];
    if (MODE == MODE_PERIODIC) {
      const long long iyp = (y + 1 == ny) ? idx - (ny - 1) : idx + 1;
      const long long ixp = (x + 1 == nx) ? (long long)y : idx + ny;
      p.hx[idx] = fsub(p.hx[idx], fmul(p.a, fsub(p.ez[iyp], e)));
      p.hy[idx] = fadd(p.hy[idx], fmul(p.a, fsub(p.ez[ixp], e)));
    } else {
      if (y < ny - 1) p.hx[idx] = fsub(p.hx[idx], fmul(p.a, fsub(p.ez[idx + 1], e)));
      if (x < nx - 1) p.hy[idx] = fadd(p.hy[idx], fmul(p.a, fsub(p.ez[idx + ny], e)));
    }
  }
}

__device__ __forceinline__ float add_line_sources(const Step2D& p, int y, float v) {
  for (int s = 0; s < p.n_src; ++s) {
    if (p.src_y[s] == y)
      v = fadd(v, fmul(p.src_amp[s], p.wave[(long long)p.src_wave[s] * p.wave_len + p.step]));
  }
  return v;
}

__device__ __forceinline__ bool in_wall(const Step2D& p, int x, int y) {
  for (int w = 0; w < p.n_wall; ++w) {
    if (p.wall_y[w] == y) {
      const int g0 = p.wall_g0[w], g1 = p.wall_g1[w];
      if (g0 < 0 || x < g0 || x >= g1) return true;
    }
  }
  return false;
}

// E update.  FUSE_POST: damping, sources and conductors in the same pass
// (ABSORBING, where no edge rule runs between them).
template <int MODE, bool FUSE_POST>
__global__ void __launch_bounds__(256) k2d_e(const __grid_constant__ Step2D p) {
  const int nx = p.nx, ny = p.ny;
  const long long n = (long long)nx * ny;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(idx % ny);
    const int x = (int)(idx / ny);
    float e = p.ez[idx];
    if (MODE == MODE_PERIODIC) {
      const long long ixm = (x == 0) ? idx + (long long)(nx - 1) * ny : idx - ny;
      const long long iym = (y == 0) ? idx + (ny - 1) : idx - 1;
      const float dhy = fsub(p.hy[idx], p.hy[ixm]);
      const float dhx = fsub(p.hx[idx], p.hx[iym]);
      e = fadd(e, fmul(p.b, fsub(dhy, dhx)));
    } else if (x >= 1 && y >= 1) {
      const float dhy = fsub(p.hy[idx], p.hy[idx - ny]);
      const float dhx = fsub(p.hx[idx], p.hx[idx - 1]);
      e = fadd(e, fmul(p.b, fsub(dhy, dhx)));
    }
    if (FUSE_POST) {
      if (MODE == MODE_ABSORB) e = fmul(e, fmul(__ldg(p.damp[0] + x), __ldg(p.damp[1] + y)));
      e = add_line_sources(p, y, e);
      if (in_wall(p, x, y)) e = 0.0f;
    }
    p.ez[idx] = e;
  }
}

// Edge rules (periodic: wrap, reflecting: mirror) for Ez, Hx, Hy in the
// reference's order (rows 0 and nx-1, then columns 0 and ny-1, so the column
// copies see the row copies), then sources, then conductors.  One block.
template <int MODE>
__global__ void __launch_bounds__(1024) k2d_post(const __grid_constant__ Step2D p) {
  const int nx = p.nx, ny = p.ny;
  const int t = threadIdx.x, nt = blockDim.x;
  const bool per = (MODE == MODE_PERIODIC);
  float* fs[3] = {p.ez, p.hx, p.hy};
  // f[0,:] = f[-2,:] (periodic) / f[1,:] (reflecting)
  for (int c = 0; c < 3; ++c) {
    float* f = fs[c];
    for (int j = t; j < ny; j += nt) f[j] = per ? f[(long long)(nx - 2) * ny + j] : f[(long long)ny + j];
  }
  __syncthreads();
  // f[-1,:] = f[1,:] (periodic) / f[-2,:] (reflecting)
  for (int c = 0; c < 3; ++c) {
    float* f = fs[c];
    for (int j = t; j < ny; j += nt)
      f[(long long)(nx - 1) * ny + j] = per ? f[(long long)ny + j] : f[(long long)(nx - 2) * ny + j];
  }
  __syncthreads();
  // f[:,0] = f[:,-2] / f[:,1]
  for (int c = 0; c < 3; ++c) {
    float* f = fs[c];
    for (int i = t; i < nx; i += nt) {
      const long long r = (long long)i * ny;
      f[r] = per ? f[r + ny - 2] : f[r + 1];
    }
  }
  __syncthreads();
  // f[:,-1] = f[:,1] / f[:,-2]
  for (int c = 0; c < 3; ++c) {
    float* f = fs[c];
    for (int i = t; i < nx; i += nt) {
      const long long r = (long long)i * ny;
      f[r + ny - 1] = per ? f[r + 1] : f[r + ny - 2];
    }
  }
  __syncthreads();
  // sources over whole rows, then conductors
  for (int i = t; i < nx; i += nt) {
    for (int s = 0; s < p.n_src; ++s) {
      const long long idx = (long long)i * ny + p.src_y[s];
      p.ez[idx] = fadd(p.ez[idx],
                       fmul(p.src_amp[s], p.wave[(long long)p.src_wave[s] * p.wave_len + p.step]));
    }
  }
  __syncthreads();
  for (int i = t; i < nx; i += nt) {
    for (int w = 0; w < p.n_wall; ++w) {
      const int g0 = p.wall_g0[w], g1 = p.wall_g1[w];
      if (g0 < 0 || i < g0 || i >= g1) p.ez[(long long)i * ny + p.wall_y[w]] = 0.0f;
    }
  }
}

// ---------------------------------------------------------------------------
// several steps per launch
// ---------------------------------------------------------------------------
//
// A block owns a tile of rows (x) and columns (y) and keeps the tile with a
// halo of `halo` cells on every side (the window: W columns by NS * R rows)
// in registers and shared memory for `steps` steps: a step takes one cell of
// validity off each side of the window, so after `steps` steps the tile is
// exact.  Blocks recompute each other's cells with the same operations, so
// the values equal the one-step kernels' bit for bit.  Reads come from one
// buffer set and the tile goes to the other (and to a saved frame).
//
// A thread owns R consecutive rows of two columns: its cells, their row
// neighbours and one column neighbour each are registers; the other column
// and the rows of the next strip go through shared memory, even and odd
// columns in arrays of their own (no bank conflicts).  Two barriers a step;
// five in the windows that hold the wrapped or mirrored edge rows and columns,
// whose copies read cells of other threads.  Windows without an edge, a
// damping layer or such copies run code without their conditions.
//
// Why: a step of the kernels above is two or three launches with nothing to do
// for most of the chip (200 x 200: 2.1 and 2.6 us of kernels, 9.7 us a step
// with the host's launches; the edge copies of one block add 7.4 us).  Here a
// small grid is bound by the latency of a window's barriers and shared-memory
// reads (about 0.5 us a step), a large one by instruction issue.  Measured per
// step on one B200, before and after: 200 x 200 absorbing 9.7 and 0.91 us,
// 151 x 203 mirrored 18 and 1.5 us, 1024 x 1024 absorbing 17 and 3.4 us.
struct Block2D {
  Step2D p;            // step: the first one; fields unused
  const float* in[3];  // Ez, Hx, Hy
  float* out[3];
  float* frame[3];     // saved frame, or null
  int steps, halo;
};

constexpr int B2D_MAX_STEPS = 16;
constexpr int B2D_MAX_SRC = 16;  // line sources whose samples a block keeps

// Window of W columns by NS * R rows, W / 2 * NS threads.
template <int W, int NS, int R>
struct B2DLayout {
  static constexpr int ROWS = NS * R, NT = W / 2 * NS;
  static constexpr int HALF = (ROWS + 1) * (W / 2);  // one array of one column parity
  static constexpr int FLOATS = 6 * HALF + B2D_MAX_STEPS * B2D_MAX_SRC;
  static constexpr size_t SMEM_BYTES = sizeof(float) * (size_t)FLOATS;
};

// MODE: MODE_ABSORB, MODE_PERIODIC or MODE_PEC (mirrored edges).
template <int MODE, int W, int NS, int R>
__global__ void __launch_bounds__(W / 2 * NS, 1024 / (W / 2 * NS))
    k2d_steps(const __grid_constant__ Block2D b) {
  using L = B2DLayout<W, NS, R>;
  constexpr int ROWS = L::ROWS, NT = L::NT, HW = W / 2;
  constexpr bool PER = MODE == MODE_PERIODIC, POST = MODE != MODE_ABSORB;
  extern __shared__ float smem2d[];
  float* const E = smem2d;            // [column parity][ROWS + 1][W / 2]
  float* const HX = E + 2 * L::HALF;
  float* const HY = HX + 2 * L::HALF;  // row i holds Hy of row i - 1
  float* const SV = HY + 2 * L::HALF;  // source samples [step][source]
  const Step2D& p = b.p;
  const int nx = p.nx, ny = p.ny;
  const int tid = threadIdx.x;
  const int l = tid % HW, i0 = (tid / HW) * R;
  const int th = ROWS - 2 * b.halo, tw = W - 2 * b.halo;
  const int tx0 = blockIdx.y * th, ty0 = blockIdx.x * tw;  // tile
  const int x0 = tx0 - b.halo, y0 = ty0 - b.halo;          // window
#define AT(A, c, i, m) A[(c) * L::HALF + (i) * HW + (m)]

  grid_dep_wait();
  grid_dep_launch_dependents();
  const bool sv = p.n_src <= B2D_MAX_SRC;
  if (sv) {
    for (int t = tid; t < b.steps * p.n_src; t += NT) {
      const int k = t / p.n_src, q = t - k * p.n_src;
      SV[t] = fmul(p.src_amp[q], p.wave[(long long)p.src_wave[q] * p.wave_len + p.step + k]);
    }
  }
  // the cells; update conditions, conductors, edge rows and owned cells as bit
  // masks over r * 2 + c
  float e[R][2], hx[R][2], hy[R][2], dx[R], dy[2];
  int gy[2];
  unsigned m_hy = 0, m_e = 0, m_wall = 0, m_top = 0, m_bot = 0, m_own = 0;
  unsigned m_src = 0, m_lo = 0, m_hi = 0;  // per column
  bool u_hx[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    gy[c] = y0 + 2 * l + c;
    if (PER) gy[c] = ((gy[c] % ny) + ny) % ny;
    u_hx[c] = PER || gy[c] < ny - 1;
    for (int q = 0; q < p.n_src; ++q)
      if (p.src_y[q] == gy[c]) m_src |= 1u << c;
    if (POST && gy[c] == 0) m_lo |= 1u << c;
    if (POST && gy[c] == ny - 1) m_hi |= 1u << c;
    dy[c] = MODE == MODE_ABSORB && gy[c] >= 0 && gy[c] < ny ? __ldg(p.damp[1] + gy[c]) : 1.0f;
  }
  bool special = !u_hx[0] || !u_hx[1];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    int gx = x0 + i0 + r;
    const bool own_row = i0 + r >= b.halo && i0 + r < b.halo + th && gx < nx;
    if (PER) gx = ((gx % nx) + nx) % nx;
    dx[r] = MODE == MODE_ABSORB && gx >= 0 && gx < nx ? __ldg(p.damp[0] + gx) : 1.0f;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const unsigned bit = 1u << (2 * r + c);
      const int j = 2 * l + c;
      const bool in = gx >= 0 && gx < nx && gy[c] >= 0 && gy[c] < ny;
      if (own_row && j >= b.halo && j < b.halo + tw && y0 + j < ny) m_own |= bit;
      const long long g = (long long)gx * ny + gy[c];
      e[r][c] = in ? b.in[0][g] : 0.0f;
      hx[r][c] = in ? b.in[1][g] : 0.0f;
      hy[r][c] = in ? b.in[2][g] : 0.0f;
      if (PER || gx < nx - 1) m_hy |= bit;
      if (PER || (gx >= 1 && gy[c] >= 1)) m_e |= bit;
      if (in && in_wall(p, gx, gy[c])) m_wall |= bit;
      if (POST && in && gx == 0) m_top |= bit;
      if (POST && in && gx == nx - 1) m_bot |= bit;
      if (MODE == MODE_ABSORB && fmul(dx[r], dy[c]) != 1.0f) special = true;
      AT(E, c, i0 + r, l) = e[r][c];
      AT(HX, c, i0 + r, l) = hx[r][c];
      AT(HY, c, i0 + r + 1, l) = hy[r][c];
    }
  }
  for (int t = tid; t < HW; t += NT)
#pragma unroll
    for (int c = 0; c < 2; ++c) AT(E, c, ROWS, t) = AT(HX, c, ROWS, t) = AT(HY, c, 0, t) = 0.0f;
  constexpr unsigned ALL = (1u << (2 * R)) - 1u;
  special = special || m_hy != ALL || m_e != ALL;
  // windows with an edge row or column to copy, an update condition or damping
  // (the same in every thread of the block)
  const bool post = __syncthreads_or(POST && (m_top | m_bot | m_lo | m_hi));
  special = __syncthreads_or(special);
  const int lr = min(l + 1, HW - 1), ll = max(l - 1, 0);
  const float ca = p.a, cbe = p.b;

  auto sources_walls = [&](int k) {
    if (m_src) {
      for (int q = 0; q < p.n_src; ++q) {
        const int y = p.src_y[q];
        if (y != gy[0] && y != gy[1]) continue;
        const float v = sv ? SV[k * p.n_src + q]
                           : fmul(p.src_amp[q],
                                  p.wave[(long long)p.src_wave[q] * p.wave_len + p.step + k]);
#pragma unroll
        for (int c = 0; c < 2; ++c)
          if (y == gy[c])
#pragma unroll
            for (int r = 0; r < R; ++r) e[r][c] = fadd(e[r][c], v);
      }
    }
    if (m_wall) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          if ((m_wall >> (2 * r + c)) & 1u) e[r][c] = 0.0f;
    }
  };
  // H and E updates of a step (a barrier between them); SP: with the update
  // conditions and damping
  auto update = [&](auto sp_c) {
    constexpr bool SP = decltype(sp_c)::value;
    const float en[2] = {AT(E, 0, i0 + R, l), AT(E, 1, i0 + R, l)};
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float right = AT(E, 0, i0 + r, lr);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float er = c == 0 ? e[r][1] : right;
        const float ed = r + 1 < R ? e[(r + 1) % R][c] : en[c];
        if (!SP || u_hx[c]) hx[r][c] = fsub(hx[r][c], fmul(ca, fsub(er, e[r][c])));
        if (!SP || ((m_hy >> (2 * r + c)) & 1u))
          hy[r][c] = fadd(hy[r][c], fmul(ca, fsub(ed, e[r][c])));
      }
      AT(HX, 1, i0 + r, l) = hx[r][1];
    }
    AT(HY, 0, i0 + R, l) = hy[R - 1][0];
    AT(HY, 1, i0 + R, l) = hy[R - 1][1];
    __syncthreads();
    const float hp[2] = {AT(HY, 0, i0, l), AT(HY, 1, i0, l)};
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float left = AT(HX, 1, i0 + r, ll);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float d = fsub(fsub(hy[r][c], r > 0 ? hy[(r + R - 1) % R][c] : hp[c]),
                             fsub(hx[r][c], c == 0 ? left : hx[r][0]));
        if (!SP || ((m_e >> (2 * r + c)) & 1u)) e[r][c] = fadd(e[r][c], fmul(cbe, d));
        if (SP && MODE == MODE_ABSORB) e[r][c] = fmul(e[r][c], fmul(dx[r], dy[c]));
      }
    }
  };
  // what the neighbours read of E: the even column, and the strip's first row
  auto put_e = [&] {
#pragma unroll
    for (int r = 0; r < R; ++r) AT(E, 0, i0 + r, l) = e[r][0];
    AT(E, 1, i0, l) = e[0][1];
  };

  for (int k = 0; k < b.steps; ++k) {
    if (special) update(BoolC<true>{});
    else update(BoolC<false>{});
    if (!post) {
      sources_walls(k);
      put_e();
      __syncthreads();
      continue;
    }
    // edge rules of Ez, Hx, Hy: rows 0 and nx-1, then columns 0 and ny-1 (the
    // column copies see the row copies), then sources, then conductors
    // (the odd columns of Hx and the strip's last row of Hy are there already)
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        AT(E, c, i0 + r, l) = e[r][c];
        if (c == 0) AT(HX, c, i0 + r, l) = hx[r][c];
        if (r + 1 < R) AT(HY, c, i0 + r + 1, l) = hy[r][c];
      }
    __syncthreads();
    if (m_top | m_bot) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const bool top = (m_top >> (2 * r + c)) & 1u, bot = (m_bot >> (2 * r + c)) & 1u;
          if (!top && !bot) continue;
          // (a source row outside the window belongs to a cell that is no
          // longer valid; the index is clamped)
          const int i = min(max(i0 + r + (PER ? (top ? -2 : 2) : (top ? 1 : -1)), 0), ROWS - 1);
          AT(E, c, i0 + r, l) = e[r][c] = AT(E, c, i, l);
          AT(HX, c, i0 + r, l) = hx[r][c] = AT(HX, c, i, l);
          AT(HY, c, i0 + r + 1, l) = hy[r][c] = AT(HY, c, i + 1, l);
        }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const bool lo = (m_lo >> c) & 1u, hi = (m_hi >> c) & 1u;
      if (!lo && !hi) continue;
      const int j = min(max(2 * l + c + (PER ? (lo ? -2 : 2) : (lo ? 1 : -1)), 0), W - 1);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        e[r][c] = AT(E, j & 1, i0 + r, j >> 1);
        hx[r][c] = AT(HX, j & 1, i0 + r, j >> 1);
        hy[r][c] = AT(HY, j & 1, i0 + r + 1, j >> 1);
      }
    }
    __syncthreads();
    sources_walls(k);
    put_e();
    __syncthreads();
  }

#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!((m_own >> (2 * r + c)) & 1u)) continue;
      const long long g = (long long)(x0 + i0 + r) * ny + (y0 + 2 * l + c);
      b.out[0][g] = e[r][c];
      b.out[1][g] = hx[r][c];
      b.out[2][g] = hy[r][c];
      if (b.frame[0] != nullptr) {
        b.frame[0][g] = e[r][c];
        b.frame[1][g] = hx[r][c];
        b.frame[2][g] = hy[r][c];
      }
    }
#undef AT
}

}  // namespace jxf
