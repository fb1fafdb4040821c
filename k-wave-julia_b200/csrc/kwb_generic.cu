// The passes of a time step for any line length: FFTs in place in shared memory.
//
// A CTA holds L complex lines of N points in shared memory (two real lines travel as one complex
// line).  A transform is two to four stages of radix-R butterflies (R = 2 ... 16, the fewest stages
// the length allows, FftPlan): decimation in frequency forwards, its mirror image backwards.  Each
// butterfly reads and writes the same R slots, so a stage needs one buffer and one barrier; the
// last forward stage of a convolution, the multiply by its operator and the first backward stage
// run as one (conv_lines).  Between the two directions the spectrum stands in digit-reversed order.
//
// What bounds these passes is instruction fetch: a radix body is some 300 unrolled instructions,
// run by few warps.  So there is one copy of each body for all kernels of this file (the noinline
// stage functions), used for every stage of every transform, and everything that touches global
// memory is a rolled loop over elements, two in flight a thread.  Stages fused with the field
// updates (one unrolled body a radix and update) waited on instructions for 9 of 16 issue slots at
// 120 x 108 x 100 and took 154 us a step; Stockham stages of radix 2, 3, 4, 5, 7 and 8, one sweep and
// barrier a prime factor, 206 us; these take 111 us (810 x 450: 102 -> 63 us), three CTAs of up to 256
// threads an SM.
#include <algorithm>

#include "kwb_fft.cuh"
#include "kwb_record.cuh"
#include "kwb_tiles.cuh"

namespace kwb {
namespace {

// ---- stages

// The lines in shared memory: position pos of line l in slot pos + (pos >> sk), at X[slot * PL + l].
// The last radix is 2^sk, so that a stage's butterflies still lie a constant number of slots apart: every
// other stride is a multiple of it.  Without gaps (sk = 31) slot and position are the same; those lengths
// have code of their own, since the shifts cost them up to 5% (a 1-D step of 243 points 8.5 -> 9.1 us).
template <bool GAPS>
struct Lines {
  float2 *X;
  const float2 *tw;
  int L, PL, sk;
  FastDiv dL;
  __device__ __forceinline__ int slot(int pos) const { return GAPS ? pos + (pos >> sk) : pos; }
  __device__ __forceinline__ float2 &at(int l, int pos) const { return X[slot(pos) * PL + l]; }
};

// call op with the radix as a compile-time constant
template <class Op>
__device__ __forceinline__ void radix_switch(int R, Op &&op) {
  switch (R) {
    case 1: op(std::integral_constant<int, 1>{}); break;
    case 2: op(std::integral_constant<int, 2>{}); break;
    case 3: op(std::integral_constant<int, 3>{}); break;
    case 4: op(std::integral_constant<int, 4>{}); break;
    case 5: op(std::integral_constant<int, 5>{}); break;
    case 6: op(std::integral_constant<int, 6>{}); break;
    case 7: op(std::integral_constant<int, 7>{}); break;
    case 8: op(std::integral_constant<int, 8>{}); break;
    case 9: op(std::integral_constant<int, 9>{}); break;
    case 10: op(std::integral_constant<int, 10>{}); break;
    case 11: op(std::integral_constant<int, 11>{}); break;
    case 12: op(std::integral_constant<int, 12>{}); break;
    case 13: op(std::integral_constant<int, 13>{}); break;
    case 15: op(std::integral_constant<int, 15>{}); break;
    default: op(std::integral_constant<int, 16>{}); break;
  }
}

// One stage in place on all lines: butterflies of R slots st positions apart (nb of them over the
// lines, dst divides by st), twiddle table step ts.  Forward: DFT, then twiddles; backward: conjugate
// twiddles, then the inverse DFT.
template <bool INV, bool GAPS>
__device__ __noinline__ void stage(Lines<GAPS> ln, int R_, int st, int ts, int nb, FastDiv dst) {
  radix_switch(R_, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    if constexpr (R == 1) return;  // (lengths of one stage begin with a 1)
    const int step = ln.slot(st) * ln.PL;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
      const int j = fdiv(b, ln.dL), l = b - j * ln.L;
      const int blk = fdiv(j, dst), u = j - blk * st;
      float2 *x = ln.X + ln.slot(blk * st * R + u) * ln.PL + l;
      float2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = x[r * step];
      if (!INV) dft_any<R, false>(v);
      if (st > 1) {
        const int k = u * ts;
#pragma unroll
        for (int q = 1; q < R; ++q) {
          float2 c = ln.tw[q * k];
          if (INV) c.y = -c.y;
          v[q] = cmul(v[q], c);
        }
      }
      if (INV) dft_any<R, true>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) x[r * step] = v[r];
    }
  });
}

// The last forward stage, the multiply by g (digit-reversed order) and the first backward stage.  A line
// of one point has radix 1 here too: its transforms are nothing, but g still multiplies it.
template <bool GAPS>
__device__ __noinline__ void stage_top(Lines<GAPS> ln, int R_, int nb, const float2 *__restrict__ g) {
  radix_switch(R_, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
      const int j = fdiv(b, ln.dL), l = b - j * ln.L;
      float2 *x = ln.X + ln.slot(j * R) * ln.PL + l;
      float2 v[R], m[R];
#pragma unroll
      for (int r = 0; r < R; ++r) m[r] = __ldg(g + j * R + r);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = x[r * ln.PL];
      dft_any<R, false>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = cmul(v[r], m[r]);
      dft_any<R, true>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) x[r * ln.PL] = v[r];
    }
  });
}

template <bool INV, bool GAPS>
__device__ __forceinline__ void run_stage(const Lines<GAPS> &ln, const FftPlan &pl, int s) {
  stage<INV>(ln, pl.radix[s], pl.stride[s], pl.tstride[s], ln.L * pl.nbf[s], pl.div_st[s]);
  __syncthreads();
}

// Transforms of all lines, natural order <-> digit-reversed order, and circular convolution with the
// kernel whose transform is g (digit-reversed). The lines are filled before and read after; all
// threads call them.
template <bool GAPS>
__device__ __forceinline__ void fwd_lines(const Lines<GAPS> &ln, const FftPlan &pl) {
  __syncthreads();
  for (int s = 0; s < pl.nstages; ++s) run_stage<false>(ln, pl, s);
}
template <bool GAPS>
__device__ __forceinline__ void inv_lines(const Lines<GAPS> &ln, const FftPlan &pl) {
  __syncthreads();
  for (int s = pl.nstages - 1; s >= 0; --s) run_stage<true>(ln, pl, s);
}
template <bool GAPS>
__device__ __forceinline__ void conv_lines(const Lines<GAPS> &ln, const FftPlan &pl, const float2 *g) {
  const int top = pl.nstages - 1;
  __syncthreads();
  for (int s = 0; s < top; ++s) run_stage<false>(ln, pl, s);
  stage_top(ln, pl.radix[top], ln.L * pl.nbf[top], g);
  __syncthreads();
  for (int s = top - 1; s >= 0; --s) run_stage<true>(ln, pl, s);
}

// zero the padding of a convolution longer than the line
template <bool GAPS>
__device__ __forceinline__ void clear_tail(const Lines<GAPS> &ln, const FftPlan &pl) {
  for (int e = threadIdx.x + pl.n * ln.L; e < pl.m * ln.L; e += blockDim.x) {
    const int pos = fdiv(e, ln.dL);
    ln.at(e - pos * ln.L, pos) = make_float2(0.f, 0.f);
  }
}

// digit-reversed position of frequency k
__device__ __forceinline__ int pos_of(const FftPlan &pl, int k) {
  int pos = 0;
  for (int s = 0; s < pl.nstages; ++s) {
    const int q = fdiv(k, pl.div_r[s]);
    pos += (k - q * pl.radix[s]) * pl.stride[s];
    k = q;
  }
  return pos;
}

// Dynamic shared memory of a pass: the lines, the twiddles and, for passes that index the spectrum,
// the digit-reversed position of each frequency (natural order with a convolution in its place).
template <bool GAPS>
struct PassSmem {
  Lines<GAPS> ln;
  unsigned short *at_k;
};
template <bool GAPS>
__device__ __forceinline__ PassSmem<GAPS> pass_smem(const FftPlan &pl, const float2 *tw_table, int L, FastDiv dL, bool spectrum) {
  extern __shared__ float4 smem_raw[];
  const int M = fft_len(pl), PL = lines_pitch(L);
  float2 *X = reinterpret_cast<float2 *>(smem_raw), *tw = X + line_slots(pl) * PL;
  load_twiddles(tw, tw_table, M);
  PassSmem<GAPS> s{{X, tw, L, PL, pl.sk, dL}, reinterpret_cast<unsigned short *>(tw + M)};
  if (spectrum)
    for (int k = threadIdx.x; k < pl.n; k += blockDim.x)
      s.at_k[k] = (unsigned short)(pl.m > 0 ? k : pl.posof ? __ldg(pl.posof + k) : pos_of(pl, k));
  return s;
}

// Elements of the tile, UNROLL (or U) a thread at a time: load(j, l, i) for each, then use(j, l, i). Element
// i of line l; neighbouring lanes take neighbouring positions (BYROW) or lines.  A thread's last
// round may repeat its first element's load.  (810 x 450 / 120 x 108 x 100, us a step: unrolled once
// 69.6 / 116.8, twice 66.3 / 112, three times 67.0 / 113.2, four times 68.7 / 113.6, eight 83.7 / 128.)
constexpr int UNROLL = 2;
template <bool BYROW, int U = UNROLL, class Load, class Use>
__device__ __forceinline__ void elements(int L, int n, FastDiv dL, FastDiv dn, Load &&load, Use &&use) {
  const int total = L * n;
  auto split = [&](int e, int &l, int &i) {
    if (BYROW) {
      l = fdiv(e, dn);
      i = e - l * n;
    } else {
      i = fdiv(e, dL);
      l = e - i * L;
    }
  };
  for (int e0 = threadIdx.x; e0 < total; e0 += U * blockDim.x) {
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int e = e0 + j * (int)blockDim.x;
      int l, i;
      split(e < total ? e : e0, l, i);
      load(j, l, i);
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int e = e0 + j * (int)blockDim.x;
      if (e >= total) break;
      int l, i;
      split(e, l, i);
      use(j, l, i);
    }
  }
}

// The two real lines of pair l of a tile at position i (0 where a line lies past the grid's edge).
template <bool CONTIG>
struct Pairs {
  Tile T;
  int Nx;
  bool even;  // strided pairs load as one float2
  __device__ __forceinline__ Pairs(const SimDev &S, int axis, int L)
      : T(CONTIG ? tile_x(S, 2 * L, blockIdx.x) : tile_yz(S, axis, 2 * L, blockIdx.x)),
        Nx(S.N[0]),
        even(!CONTIG && (S.N[0] & 1) == 0) {}
  __device__ __forceinline__ int step() const { return CONTIG ? Nx : 1; }
  __device__ __forceinline__ long long off(int l, int i) const {
    return CONTIG ? T.base + (long long)(2 * l) * Nx + i : T.base + (long long)i * T.stride + 2 * l;
  }
  __device__ __forceinline__ float2 load(const float *f, int l, int i) const {
    const float *a = f + off(l, i);
    const int n = T.cnt - 2 * l;
    if (even && n >= 2) return __ldcg(reinterpret_cast<const float2 *>(a));
    return make_float2(n > 0 ? __ldcg(a) : 0.f, n > 1 ? __ldcg(a + step()) : 0.f);
  }
  __device__ __forceinline__ void store(float *f, int l, int i, float2 v) const {
    float *a = f + off(l, i);
    const int n = T.cnt - 2 * l;
    if (even && n >= 2) {
      *reinterpret_cast<float2 *>(a) = v;
      return;
    }
    if (n > 0) a[0] = v.x;
    if (n > 1) a[step()] = v.y;
  }
  // v with the lines past the edge at zero
  __device__ __forceinline__ float2 live(int l, float2 v) const {
    const int n = T.cnt - 2 * l;
    return make_float2(n > 0 ? v.x : 0.f, n > 1 ? v.y : 0.f);
  }
};

// ---- line pass

// Gradient, field update, gradient, field update of one tile of 2L lines.  The first pass of a step
// (y) waits for the pressure its predecessor wrote; the others load theirs before they wait (as
// k_line_fast).
template <bool CONTIG, bool GAPS>
__global__ void __launch_bounds__(KWB_PASS_THREADS_MAX, 3)
    k_line_pass(const __grid_constant__ SimDev S, int axis, int mode, FastDiv dL, long long step_s) {
  const FftPlan &pl = S.plan[axis];
  const int N = pl.n, L = S.L_line[axis];
  const Lines<GAPS> ln = pass_smem<GAPS>(pl, S.tw[axis], L, dL, false).ln;
  const Pairs<CONTIG> pr(S, axis, L);
  const Tile &T = pr.T;
  // point sources on the tile's lines: a thread fetches the entry it will apply ahead of time
  const bool step = mode == KWB_MODE_STEP;
  int uq0 = 0, un = 0, pq0 = 0, pn = 0;
  SrcEntry ue{}, pe{};
  if (step && S.u_sig[axis] && S.u_line_ptr[axis]) {
    uq0 = S.u_line_ptr[axis][T.first_line];
    un = S.u_line_ptr[axis][T.first_line + T.cnt] - uq0;
    if ((int)threadIdx.x < un) ue = S.u_entry[axis][uq0 + threadIdx.x];
  }
  if (step && S.n_p > 0 && S.p_line_ptr[axis]) {
    pq0 = S.p_line_ptr[axis][T.first_line];
    pn = S.p_line_ptr[axis][T.first_line + T.cnt] - pq0;
    if ((int)threadIdx.x < pn) pe = S.p_entry[axis][pq0 + threadIdx.x];
  }
  const bool wait_first = !step || axis == 1 || S.ndim == 1;
  if (wait_first) KWB_STEP_KERNEL_PROLOGUE();
  const long long t = step_index(S, step_s);
  float uval = 0.f, pval = 0.f;
  const int tcol_u = S.u_sig[axis] ? (int)(min(t + 1, (long long)S.u_cols[axis]) - 1) : 0;
  const int tcol_p = (int)(min(t + 1, (long long)S.p_cols) - 1);
  if ((int)threadIdx.x < un) uval = S.u_sig[axis][(long long)tcol_u * S.n_u + ue.j];
  if ((int)threadIdx.x < pn) pval = S.p_sig[(long long)tcol_p * S.n_p + pe.j];
  const float2 zero = make_float2(0.f, 0.f);
  float2 a[UNROLL], b[UNROLL], c[UNROLL];
  float d[UNROLL];

  // d/dx_d p  (staggered +)
  elements<CONTIG>(L, N, dL, pl.div_n, [&](int j, int l, int i) { a[j] = pr.load(S.p, l, i); },
                   [&](int j, int l, int i) { ln.at(l, i) = a[j]; });
  clear_tail(ln, pl);
  if (!wait_first) KWB_STEP_KERNEL_PROLOGUE();
  if (step && t >= S.Nt) return;
  twiddles_landed();
  conv_lines(ln, pl, S.gdif[axis][0]);

  // velocity update u = pml_sg (pml_sg u - dt/rho_sg dp), with pml = 1 - deficit
  float *__restrict__ ud = S.u[axis];
  float *__restrict__ rd = S.rho[axis];
  const float *__restrict__ rho0 = S.rho0;
  elements<CONTIG>(
      L, N, dL, pl.div_n,
      [&](int j, int l, int i) {
        a[j] = step ? pr.load(ud, l, i) : zero;
        b[j] = rho0 ? pr.load(rho0, l, i) : zero;
        c[j] = rho0 ? pr.load(rho0, l, i + 1 == N ? 0 : i + 1) : zero;  // periodic neighbour
        d[j] = __ldg(S.pml_sg_def[axis] + i);
      },
      [&](int j, int l, int i) {
        const float2 g = ln.at(l, i);
        float2 coef = make_float2(S.dt_over_rho0_s, S.dt_over_rho0_s), v;
        if (rho0) coef = make_float2(S.dt / (0.5f * (b[j].x + c[j].x)), S.dt / (0.5f * (b[j].y + c[j].y)));
        if (!step) {
          // u(-dt/2) = -dt/(2 rho_sg) dp0  (first_order_steps.jl:128-136)
          v = make_float2(-0.5f * coef.x * g.x, -0.5f * coef.y * g.y);
        } else {
          v = make_float2(fmaf(-d[j], a[j].x, a[j].x), fmaf(-d[j], a[j].y, a[j].y));
          v = make_float2(fmaf(-coef.x, g.x, v.x), fmaf(-coef.y, g.y, v.y));
          v = make_float2(fmaf(-d[j], v.x, v.x), fmaf(-d[j], v.y, v.y));
        }
        pr.store(ud, l, i, v);
        ln.at(l, i) = pr.live(l, v);
      });
  if (!step) {
    // rho_d = p0 / (D c0^2)   (first_order_steps.jl:77, 117-118, 165-167)
    elements<CONTIG>(
        L, N, dL, pl.div_n,
        [&](int j, int l, int i) {
          a[j] = pr.load(S.p, l, i);
          b[j] = S.c0sq ? pr.load(S.c0sq, l, i) : make_float2(S.c0sq_s, S.c0sq_s);
        },
        [&](int j, int l, int i) {
          pr.store(rd, l, i, make_float2(a[j].x / ((float)S.D * b[j].x), a[j].y / ((float)S.D * b[j].y)));
        });
    return;
  }
  // velocity sources on the lines of this tile (first_order_steps.jl:586-617, 646-690)
  if (un > 0) {
    __syncthreads();
    for (int q = threadIdx.x; q < un; q += blockDim.x) {
      if (q != (int)threadIdx.x) {
        ue = S.u_entry[axis][uq0 + q];
        uval = S.u_sig[axis][(long long)tcol_u * S.n_u + ue.j];
      }
      const int col = ue.line - T.first_line;
      float *cell = reinterpret_cast<float *>(&ln.at(col >> 1, ue.pos)) + (col & 1);
      const float nv = (S.u_mode == 0) ? uval : *cell + uval;
      *cell = nv;
      ud[pr.off(col >> 1, ue.pos) + (col & 1) * pr.step()] = nv;
    }
  }

  // d/dx_d u_d  (staggered -)
  clear_tail(ln, pl);
  conv_lines(ln, pl, S.gdif[axis][1]);

  // density update rho_d = pml (pml rho_d - dt rho0 du)
  elements<CONTIG>(
      L, N, dL, pl.div_n,
      [&](int j, int l, int i) {
        a[j] = pr.load(rd, l, i);
        b[j] = rho0 ? pr.load(rho0, l, i) : zero;
        d[j] = __ldg(S.pml_def[axis] + i);
        // u as this CTA stored it, for the axisymmetric radial term
        c[j] = axis == 1 && S.inv_r ? pr.load(ud, l, i) : zero;
      },
      [&](int j, int l, int i) {
        float2 du = ln.at(l, i);
        const float2 coef = rho0 ? make_float2(S.dt * b[j].x, S.dt * b[j].y) : make_float2(S.dt_rho0_s, S.dt_rho0_s);
        if (axis == 1 && S.inv_r) {  // + u_r / r (axisymmetric.jl:183)
          const float ir = __ldg(S.inv_r + i);
          du = make_float2(fmaf(c[j].x, ir, du.x), fmaf(c[j].y, ir, du.y));
        }
        float2 v = make_float2(fmaf(-d[j], a[j].x, a[j].x), fmaf(-d[j], a[j].y, a[j].y));
        v = make_float2(fmaf(-coef.x, du.x, v.x), fmaf(-coef.y, du.y, v.y));
        pr.store(rd, l, i, make_float2(fmaf(-d[j], v.x, v.x), fmaf(-d[j], v.y, v.y)));
      });

  // pressure (mass) sources: rho_d (+)= p / (D c^2)   (first_order_steps.jl:619-640, 692-715)
  if (pn > 0) {
    __syncthreads();
    for (int q = threadIdx.x; q < pn; q += blockDim.x) {
      if (q != (int)threadIdx.x) {
        pe = S.p_entry[axis][pq0 + q];
        pval = S.p_sig[(long long)tcol_p * S.n_p + pe.j];
      }
      const int col = pe.line - T.first_line;
      float *cell = rd + pr.off(col >> 1, pe.pos) + (col & 1) * pr.step();
      *cell = (S.p_mode == 0) ? pval : __ldcg(cell) + pval;
    }
  }
}

// ---- equation of state

// x R2C of [c0^2] rho (1 + Q rho), rho = sum of the split densities, Q = BonA / (2 rho0)
// (first_order_steps.jl:236-241, 275-279); CHANGE: of its change since the last step
// (first_order_steps.jl:255-263, 436-440)
template <bool GAPS, bool CHANGE>
__global__ void __launch_bounds__(KWB_PASS_THREADS_MAX, 3)
    k_eos_x_fwd(const __grid_constant__ SimDev S, FastDiv dL, FastDiv dn1, long long step_s) {
  const FftPlan &pl = S.plan[0];
  const int N = pl.n, L = S.L_eosx, n1 = S.n1;
  const PassSmem<GAPS> sm = pass_smem<GAPS>(pl, S.tw[0], L, dL, true);
  const Lines<GAPS> &ln = sm.ln;
  const Pairs<true> pr(S, 0, L);
  KWB_STEP_KERNEL_PROLOGUE();
  if (step_index(S, step_s) >= S.Nt) return;
  const float2 zero = make_float2(0.f, 0.f);
  float2 a[UNROLL], b[UNROLL], c[UNROLL], q[UNROLL], w[UNROLL];
  elements<true>(
      L, N, dL, pl.div_n,
      [&](int j, int l, int i) {
        a[j] = pr.load(S.rho[0], l, i);
        b[j] = S.D > 1 ? pr.load(S.rho[1], l, i) : zero;
        c[j] = S.D > 2 ? pr.load(S.rho[2], l, i) : zero;
        q[j] = S.nonlinear && S.nlq ? pr.load(S.nlq, l, i) : make_float2(S.nlq_s, S.nlq_s);
        w[j] = S.c0sq ? pr.load(S.c0sq, l, i) : zero;
      },
      [&](int j, int l, int i) {
        float2 v = a[j];
        if (S.D > 1) v = cadd(v, b[j]);
        if (S.D > 2) v = cadd(v, c[j]);
        if (S.nonlinear) v = make_float2(v.x * fmaf(q[j].x, v.x, 1.0f), v.y * fmaf(q[j].y, v.y, 1.0f));
        if (S.c0sq) v = make_float2(w[j].x * v.x, w[j].y * v.y);
        if (CHANGE) {  // since the last step
          const float2 r = v;
          v = csub(v, pr.load(S.rho_prev, l, i));
          pr.store(S.rho_prev, l, i, r);
        }
        ln.at(l, i) = pl.m > 0 ? cmul(v, __ldg(pl.chirp + i)) : v;
      });
  clear_tail(ln, pl);
  twiddles_landed();
  if (pl.m > 0) conv_lines(ln, pl, pl.chirp_ft);
  else fwd_lines(ln, pl);
  // split the two packed real rows: A_k = (Z_k + conj Z_-k)/2, B_k = (Z_k - conj Z_-k)/(2i)
  for (int e = threadIdx.x; e < L * n1; e += blockDim.x) {
    const int l = fdiv(e, dn1), k = e - l * n1, km = k == 0 ? 0 : N - k;
    const long long rowa = (long long)pr.T.outer * S.N[1] + pr.T.y0 + 2 * l;
    float2 z = ln.at(l, sm.at_k[k]), zm = ln.at(l, sm.at_k[km]);
    if (pl.m > 0) {
      z = cmul(z, __ldg(pl.chirp + k));
      zm = cmul(zm, __ldg(pl.chirp + km));
    }
    const float2 A = make_float2(0.5f * (z.x + zm.x), 0.5f * (z.y - zm.y));
    const float2 B = make_float2(0.5f * (z.y + zm.y), -0.5f * (z.x - zm.x));
    if (2 * l < pr.T.cnt) S.spec[rowa * n1 + k] = A;
    if (2 * l + 1 < pr.T.cnt) S.spec[(rowa + 1) * n1 + k] = B;
  }
}

// x C2R to the pressure (mul_x: 1-D, where no other pass multiplies by M)
template <bool GAPS>
__global__ void __launch_bounds__(KWB_PASS_THREADS_MAX, 3)
    k_eos_x_inv(const __grid_constant__ SimDev S, FastDiv dL, FastDiv dn1, long long step_s, int mul_x) {
  const FftPlan &pl = S.plan[0];
  const int N = pl.n, L = S.L_eosx, n1 = S.n1;
  const PassSmem<GAPS> sm = pass_smem<GAPS>(pl, S.tw[0], L, dL, true);
  const Lines<GAPS> &ln = sm.ln;
  const Pairs<true> pr(S, 0, L);
  const bool even = (N & 1) == 0;
  KWB_STEP_KERNEL_PROLOGUE();
  if (step_index(S, step_s) >= S.Nt) return;
  __syncthreads();  // the positions
  auto bin = [&](long long q, int k) -> float2 {
    float2 v = __ldcg(S.spec + q * n1 + k);
    if (mul_x) {
      const float m = S.M[q * n1 + k];
      if (S.dispersion) {  // the spectrum of the step before (build_eos_multiplier)
        const float m2 = S.M2[q * n1 + k];
        const float2 b = __ldcg(S.spec2 + q * n1 + k);
        S.spec2[q * n1 + k] = v;
        v = make_float2(fmaf(m2, b.x, m * v.x), fmaf(m2, b.y, m * v.y));
      } else {
        v = cscale(v, m);
      }
    }
    return v;
  };
  // two rows as one line, at its digit-reversed position (Bluestein: conjugated, times the chirp, in
  // natural order)
  auto put = [&](int l, int k, float2 z) {
    if (pl.m > 0) z = cmul(make_float2(z.x, -z.y), __ldg(pl.chirp + k));
    ln.at(l, sm.at_k[k]) = z;
  };
  const float2 zero = make_float2(0.f, 0.f);
  for (int e0 = threadIdx.x; e0 < L * n1; e0 += UNROLL * blockDim.x) {
    float2 A[UNROLL], B[UNROLL];
#pragma unroll
    for (int j = 0; j < UNROLL; ++j) {
      const int e = e0 + j * (int)blockDim.x;
      const int l = fdiv(e, dn1), k = e - l * n1;
      const int n = e < L * n1 ? pr.T.cnt - 2 * l : 0;
      const long long rowa = (long long)pr.T.outer * S.N[1] + pr.T.y0 + 2 * l;
      A[j] = n > 0 ? bin(rowa, k) : zero;
      B[j] = n > 1 ? bin(rowa + 1, k) : zero;
    }
#pragma unroll
    for (int j = 0; j < UNROLL; ++j) {
      const int e = e0 + j * (int)blockDim.x;
      if (e >= L * n1) break;
      const int l = fdiv(e, dn1), k = e - l * n1;
      if (k == 0 || (even && 2 * k == N)) {
        // c2r ignores the imaginary part of the DC and Nyquist bins
        put(l, k, make_float2(A[j].x, B[j].x));
      } else {
        put(l, k, make_float2(A[j].x - B[j].y, A[j].y + B[j].x));
        put(l, N - k, make_float2(A[j].x + B[j].y, B[j].x - A[j].y));
      }
    }
  }
  clear_tail(ln, pl);
  twiddles_landed();
  if (pl.m > 0) conv_lines(ln, pl, pl.chirp_ft);
  else inv_lines(ln, pl);
  elements<true>(L, N, dL, pl.div_n, [](int, int, int) {},
                 [&](int, int l, int i) {
                   float2 z = ln.at(l, i);
                   if (pl.m > 0) {
                     z = cmul(z, __ldg(pl.chirp + i));
                     z.y = -z.y;
                   }
                   pr.store(S.p, l, i, z);
                 });
}

// y- or z-direction FFTs of the half spectrum (complex columns kx0..kx0+L-1)
template <bool GAPS>
__global__ void __launch_bounds__(KWB_PASS_THREADS_MAX, 3)
    k_spec_pass(const __grid_constant__ SimDev S, int axis, int op, FastDiv dL, long long step_s) {
  const FftPlan &pl = S.plan[axis];
  const int N = pl.n, L = S.L_spec[axis], n1 = S.n1, Ny = S.N[1];
  const PassSmem<GAPS> sm = pass_smem<GAPS>(pl, S.tw[axis], L, dL, true);
  const Lines<GAPS> &ln = sm.ln;
  const int tpp = (n1 + L - 1) / L;
  const int o = blockIdx.x / tpp;
  const int k0 = (blockIdx.x - o * tpp) * L;
  const int cnt = min(L, n1 - k0);
  const bool blue = pl.m > 0;
  // element i of line l of the spectra, and of the multipliers, which have the same layout
  const long long base = axis == 1 ? (long long)o * n1 * Ny + k0 : (long long)o * n1 + k0;
  const long long stride = axis == 1 ? n1 : (long long)n1 * Ny;
  auto at = [&](int l, int i) -> long long { return base + (long long)i * stride + l; };
  const float2 zero = make_float2(0.f, 0.f);
  float2 a[UNROLL], b[UNROLL];
  float m[UNROLL], m2[UNROLL];
  KWB_STEP_KERNEL_PROLOGUE();
  if (step_index(S, step_s) >= S.Nt) return;
  __syncthreads();  // the positions
  // Bluestein's inverse transform is the conjugate of the forward one of the conjugate
  const bool inv = op == KWB_SPEC_INV;
  elements<false>(
      L, N, dL, pl.div_n, [&](int j, int l, int i) { a[j] = l < cnt ? __ldcg(S.spec + at(l, i)) : zero; },
      [&](int j, int l, int i) {
        if (blue) ln.at(l, i) = cmul(inv ? make_float2(a[j].x, -a[j].y) : a[j], __ldg(pl.chirp + i));
        else ln.at(l, inv ? (int)sm.at_k[i] : i) = a[j];
      });
  clear_tail(ln, pl);
  twiddles_landed();
  if (blue) conv_lines(ln, pl, pl.chirp_ft);
  else if (inv) inv_lines(ln, pl);
  else fwd_lines(ln, pl);
  if (op == KWB_SPEC_FWD) {
    elements<false>(L, N, dL, pl.div_n, [](int, int, int) {},
                    [&](int, int l, int k) {
                      float2 z = ln.at(l, sm.at_k[k]);
                      if (blue) z = cmul(z, __ldg(pl.chirp + k));
                      if (l < cnt) S.spec[at(l, k)] = z;
                    });
    return;
  }
  if (op == KWB_SPEC_FWD_MUL_INV) {
    // the equation of state: times M, and with dispersion plus M2 times the spectrum of the step
    // before, which this pass keeps in spec2, or of the change since (build_eos_multiplier; what is kept
    // then is overwritten by the next step's)
    elements<false>(
        L, N, dL, pl.div_n,
        [&](int j, int l, int k) {
          const bool in = l < cnt;
          m[j] = in ? __ldg(S.M + at(l, k)) : 0.f;
          m2[j] = in && S.dispersion ? __ldg(S.M2 + at(l, k)) : 0.f;
          b[j] = in && S.dispersion ? __ldcg(S.spec2 + at(l, k)) : zero;
        },
        [&](int j, int l, int k) {
          float2 &x = ln.at(l, sm.at_k[k]);
          float2 z = x;
          const float2 w = blue ? __ldg(pl.chirp + k) : zero;
          if (blue) z = cmul(z, w);
          if (S.dispersion) {
            if (l < cnt) S.spec2[at(l, k)] = z;
            z = make_float2(fmaf(m2[j], b[j].x, m[j] * z.x), fmaf(m2[j], b[j].y, m[j] * z.y));
          } else {
            z = cscale(z, m[j]);
          }
          x = blue ? cmul(make_float2(z.x, -z.y), w) : z;
        });
    clear_tail(ln, pl);
    if (blue) conv_lines(ln, pl, pl.chirp_ft);
    else inv_lines(ln, pl);
  }
  elements<false>(L, N, dL, pl.div_n, [](int, int, int) {},
                  [&](int, int l, int i) {
                    float2 z = ln.at(l, i);
                    if (blue) {
                      z = cmul(z, __ldg(pl.chirp + i));
                      z.y = -z.y;
                    }
                    if (l < cnt) S.spec[at(l, i)] = z;
                  });
}

// ---- elastic gradients

// Directional derivatives of g.nf fields along `axis` on one tile of 2L real lines, U elements a thread in
// flight: 8 where a thread has 12 or more (long lines, one or a few a tile), whose sweeps are rounds of
// memory latency (512 x 2048: 168 -> 153 us a step), 2 elsewhere (60 x 45 with 8: 34 -> 41).
template <bool CONTIG, bool GAPS, int U>
__global__ void __launch_bounds__(KWB_PASS_THREADS_MAX, 3)
    k_el_grad(const __grid_constant__ SimDev S, int axis, const __grid_constant__ ElGrad g, FastDiv dL, long long step_s) {
  const FftPlan &pl = S.plan[axis];
  const int N = pl.n, L = S.L_line[axis];
  const Lines<GAPS> ln = pass_smem<GAPS>(pl, S.tw[axis], L, dL, false).ln;
  const Pairs<CONTIG> pr(S, axis, L);
  KWB_STEP_KERNEL_PROLOGUE();
  if (step_index(S, step_s) >= S.Nt) return;
  twiddles_landed();
  float2 a[U];
  for (int f = 0; f < g.nf; ++f) {
    const float *src = g.src[f];
    float *dst = g.dst[f];
    const bool acc = (g.acc >> f) & 1;
    elements<CONTIG, U>(L, N, dL, pl.div_n, [&](int j, int l, int i) { a[j] = pr.load(src, l, i); },
                     [&](int j, int l, int i) { ln.at(l, i) = a[j]; });
    clear_tail(ln, pl);
    conv_lines(ln, pl, S.gdif[axis][g.neg ? 1 : 0]);  // i k e^{+-i k d/2} / N
    elements<CONTIG, U>(L, N, dL, pl.div_n,
                     [&](int j, int l, int i) { a[j] = acc ? pr.load(dst, l, i) : make_float2(0.f, 0.f); },
                     [&](int j, int l, int i) {
                       const float2 v = ln.at(l, i);
                       pr.store(dst, l, i, acc ? cadd(a[j], v) : v);
                     });
    __syncthreads();  // the lines are refilled by the next field
  }
}

// ---- many time steps of a 1-D simulation in one launch of one CTA (first_order.jl:92-285)

// A 1-D grid is one line: its whole state fits one CTA's shared memory, and a step is three circular
// convolutions along it -- d/dx of p, d/dx of u, and the equation of state, whose multiplier is real
// and even, so that the inverse transform of the full spectrum is real as it stands -- with the
// field updates between them.  Launched pass by pass, a step of 512 points cost four kernels of about
// 5 us each (launch, first loads, tables), 20 us; what bounds it here is the chain of stages and
// block barriers (about 20) of the three convolutions, 9.4 us.  The steps of a launch keep p, u and
// rho in shared memory; the medium and the operator tables stay in L1.
template <bool GAPS>
__global__ void __launch_bounds__(KWB_PASS_THREADS_MAX, 3)
    k_steps_1d(const __grid_constant__ SimDev S, const __grid_constant__ Groups1D groups, long long t_first, int steps) {
  const FftPlan &pl = S.plan[0];
  const int N = pl.n;
  const PassSmem<GAPS> sm = pass_smem<GAPS>(pl, S.tw[0], 1, FastDiv{1u, 0u}, true);
  const Lines<GAPS> &ln = sm.ln;
  float *P = const_cast<float *>(reinterpret_cast<const float *>(ln.tw + N + (N + 3) / 4));
  float *U = P + N, *Rh = U + N;
  // dispersion: the last step's spectrum, or this step's of the change since and the last rho_eff
  float2 *Prev = reinterpret_cast<float2 *>(P) + (3 * N + 1) / 2;
  float *Rp = reinterpret_cast<float *>(Prev + N);
  const bool change = S.dispersion == KWB_DISP_CHANGE;
  const float *__restrict__ rho0 = S.rho0;
  auto set = [&](int i, float v) { ln.at(0, i) = make_float2(v, 0.f); };
  __syncthreads();  // the positions
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    P[i] = S.p[i];
    U[i] = S.u[0][i];
    Rh[i] = S.rho[0][i];
    if (change) {
      Rp[i] = S.rho_prev[i];
    } else if (S.dispersion) {  // spec2 holds k <= N/2; the field is real
      const float2 a = S.spec2[2 * i <= N ? i : N - i];
      Prev[sm.at_k[i]] = 2 * i <= N ? a : make_float2(a.x, -a.y);
    }
  }
  twiddles_landed();
  for (int s = 0; s < steps; ++s) {
    const long long t = t_first + s;
    // time reversal: the boundary data replaces the density at its points (first_order.jl:450-460)
    for (int j = threadIdx.x; j < S.n_tr; j += blockDim.x)
      Rh[S.tr_idx[j]] = S.tr_sig[(S.Nt - 1 - t) * S.n_tr + j];
    // velocity: u = pml_sg (pml_sg u - dt/rho_sg dp)
    for (int i = threadIdx.x; i < N; i += blockDim.x) set(i, P[i]);
    conv_lines(ln, pl, S.gdif[0][0]);
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      const float coef =
          rho0 ? S.dt / (0.5f * (__ldg(rho0 + i) + __ldg(rho0 + (i + 1 == N ? 0 : i + 1)))) : S.dt_over_rho0_s;
      const float es = __ldg(S.pml_sg_def[0] + i), u0 = U[i];
      const float t1 = fmaf(-coef, ln.at(0, i).x, fmaf(-es, u0, u0));
      U[i] = fmaf(-es, t1, t1);
      set(i, U[i]);
    }
    if (S.u_sig[0] && S.n_u > 0) {  // first_order_steps.jl:586-617
      __syncthreads();
      const long long col = min(t + 1, (long long)S.u_cols[0]) - 1;
      for (int q = threadIdx.x; q < S.n_u; q += blockDim.x) {
        const SrcEntry e = S.u_entry[0][q];
        const float val = S.u_sig[0][col * S.n_u + e.j];
        U[e.pos] = S.u_mode == 0 ? val : U[e.pos] + val;
        set(e.pos, U[e.pos]);
      }
    }
    // density: rho = pml (pml rho - dt rho0 du)
    conv_lines(ln, pl, S.gdif[0][1]);
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      const float coef = rho0 ? S.dt * __ldg(rho0 + i) : S.dt_rho0_s;
      const float e = __ldg(S.pml_def[0] + i), r0 = Rh[i];
      const float t1 = fmaf(-coef, ln.at(0, i).x, fmaf(-e, r0, r0));
      Rh[i] = fmaf(-e, t1, t1);
    }
    if (S.n_p > 0) {  // first_order_steps.jl:619-640
      __syncthreads();
      const long long col = min(t + 1, (long long)S.p_cols) - 1;
      for (int q = threadIdx.x; q < S.n_p; q += blockDim.x) {
        const SrcEntry e = S.p_entry[0][q];
        const float val = S.p_sig[col * S.n_p + e.j];
        Rh[e.pos] = S.p_mode == 0 ? val : Rh[e.pos] + val;
      }
      __syncthreads();
    }
    // equation of state (first_order_steps.jl:214-290)
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      float f = Rh[i];
      if (S.nonlinear) f = f * fmaf(S.nlq ? __ldg(S.nlq + i) : S.nlq_s, f, 1.0f);
      if (S.c0sq) f = __ldg(S.c0sq + i) * f;
      set(i, change ? f - Rp[i] : f);
      if (change) Rp[i] = f;
    }
    if (!S.dispersion) {
      conv_lines(ln, pl, S.eos1d);
    } else {
      fwd_lines(ln, pl);
      if (change) {
        for (int k = threadIdx.x; k < N; k += blockDim.x) Prev[k] = ln.at(0, k);
        __syncthreads();
        for (int i = threadIdx.x; i < N; i += blockDim.x) set(i, Rp[i]);
        fwd_lines(ln, pl);
      }
      for (int k = threadIdx.x; k < N; k += blockDim.x) {  // as k_spec_pass
        const int pos = sm.at_k[k], kk = 2 * k <= N ? k : N - k;
        const float m = __ldg(S.M + kk), m2 = __ldg(S.M2 + kk);
        const float2 z = ln.at(0, pos), b = Prev[pos];
        if (!change) Prev[pos] = z;
        ln.at(0, pos) = make_float2(fmaf(m2, b.x, m * z.x), fmaf(m2, b.y, m * z.y));
      }
      inv_lines(ln, pl);
    }
    for (int i = threadIdx.x; i < N; i += blockDim.x) P[i] = ln.at(0, i).x;
    if (groups.n > 0) {
      __syncthreads();
      for (int g = 0; g < groups.n; ++g) {
        const GroupDev &gd = *groups.g[g];
        for (long long j = threadIdx.x; j < gd.n; j += blockDim.x) {
          const long long v = gd.dense ? j : gd.idx[j];
          record_point(S, gd, t, j, P[v], [&](int) { return U[v]; });
        }
      }
    }
  }
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    S.p[i] = P[i];
    S.u[0][i] = U[i];
    S.rho[0][i] = Rh[i];
    if (change) S.rho_prev[i] = Rp[i];
    else if (S.dispersion && 2 * i <= N) S.spec2[i] = Prev[sm.at_k[i]];
  }
}

// the full-length operator of the 1-D equation of state, (M(|k|), 0)
__global__ void k_eos1d(float2 *out, const float *M, int N) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < N) out[k] = make_float2(M[2 * k <= N ? k : N - k], 0.f);
}

int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }
// a pass that indexes the spectrum also holds the positions
size_t spectrum_pass_smem(const FftPlan &pl, int L) {
  return line_pass_smem(pl, L) + (size_t)pl.n * sizeof(unsigned short);
}
size_t steps1d_smem(const SimDev &h) {
  const int N = h.N[0];
  return ((size_t)line_slots(h.plan[0]) * lines_pitch(1) + N + (N + 3) / 4 + (3 * N + 1) / 2 + (h.dispersion ? N : 0) +
          (h.dispersion == KWB_DISP_CHANGE ? (N + 1) / 2 : 0)) *
         sizeof(float2);
}

}  // namespace

size_t line_pass_smem(const FftPlan &pl, int L) {
  return ((size_t)line_slots(pl) * lines_pitch(L) + fft_len(pl)) * sizeof(float2);
}

// Threads per CTA: one butterfly of the first stage each, or, above KWB_PASS_THREADS_MAX of them,
// equal shares.
int pass_threads(const FftPlan &pl, int L, int tuned) {
  if (tuned > 0) return tuned;
  const int nb = L * pl.nbf[pl.radix[0] > 1 ? 0 : pl.nstages - 1];
  const int rounds = (nb + KWB_PASS_THREADS_MAX - 1) / KWB_PASS_THREADS_MAX;
  return std::max(32, ((nb + rounds - 1) / rounds + 31) / 32 * 32);
}

// op with the kernels of a plan: std::true_type where its lines have gaps
template <class Op>
auto by_gaps(const FftPlan &pl, Op &&op) {
  return pl.sk < 31 ? op(std::true_type{}) : op(std::false_type{});
}
cudaError_t generic_prime(const SimDev &h) {
  cudaError_t e = by_gaps(h.plan[0], [&](auto g) {
    constexpr bool G = decltype(g)::value;
    cudaError_t e2 = raise_dynamic_smem((const void *)k_line_pass<true, G>, line_pass_smem(h.plan[0], h.L_line[0]));
    const size_t eos = spectrum_pass_smem(h.plan[0], h.L_eosx);
    if (e2 == cudaSuccess) e2 = raise_dynamic_smem((const void *)k_eos_x_fwd<G, false>, eos);
    if (e2 == cudaSuccess) e2 = raise_dynamic_smem((const void *)k_eos_x_fwd<G, true>, eos);
    return e2 == cudaSuccess ? raise_dynamic_smem((const void *)k_eos_x_inv<G>, eos) : e2;
  });
  for (int a = 1; a < h.ndim && e == cudaSuccess; ++a)
    e = by_gaps(h.plan[a], [&](auto g) {
      constexpr bool G = decltype(g)::value;
      const cudaError_t e2 = raise_dynamic_smem((const void *)k_line_pass<false, G>, line_pass_smem(h.plan[a], h.L_line[a]));
      return e2 == cudaSuccess ? raise_dynamic_smem((const void *)k_spec_pass<G>, spectrum_pass_smem(h.plan[a], h.L_spec[a])) : e2;
    });
  return e;
}
// ... of a fluid pass: at least a thread for every 8 elements (first stages of radix 16 or 12 gave them 16
// or 12: 112^2 in full-width tiles, as in a batch, 82 -> 64 us a step, 360 x 240 88 -> 71, 100^3 122 -> 108),
// and where it has at most two tiles an SM and the simulation runs alone, for every 4, since its sweeps are
// then rounds of memory latency (us a step without a measured schedule: 112^2 61 -> 52, 30 x 64 37.8 -> 32.4,
// 270 x 256 63.7 -> 45.9, 810 x 450 75 -> 71); in larger grids, which hide it, so many threads leave room for
// fewer CTAs (120 x 108 x 100: 8 elements 125, 4 141).
static int fluid_threads(const SimDev &h, int axis, int L, int grid, int tuned) {
  const int thr = pass_threads(h.plan[axis], L, tuned);
  if (tuned > 0) return thr;
  const int each = h.grid_fill && grid <= 2 * h.num_sms ? 4 : 8;
  return std::max(thr, std::min(KWB_PASS_THREADS_MAX, (L * h.plan[axis].n / each + 31) / 32 * 32));
}
cudaError_t generic_line_pass(const SimDev &h, int axis, int mode, long long step_s, cudaStream_t st) {
  const int L = h.L_line[axis];
  const int grid = axis == 0 ? cdiv(h.N[1], 2 * L) * h.N[2] : cdiv(h.N[0], 2 * L) * (axis == 1 ? h.N[2] : h.N[1]);
  const int thr = fluid_threads(h, axis, L, grid, h.thr_line[axis]);
  const size_t sm = line_pass_smem(h.plan[axis], L);
  const FastDiv dL = make_fastdiv((unsigned)L);
  by_gaps(h.plan[axis], [&](auto g) {
    constexpr bool G = decltype(g)::value;
    if (axis == 0) kwb_launch(k_line_pass<true, G>, grid, thr, sm, st, h, axis, mode, dL, step_s);
    else kwb_launch(k_line_pass<false, G>, grid, thr, sm, st, h, axis, mode, dL, step_s);
  });
  return cudaGetLastError();
}
cudaError_t generic_eos(const SimDev &h, bool fwd, long long step_s, cudaStream_t st, bool change) {
  const int L = h.L_eosx, grid = cdiv(h.N[1], 2 * L) * h.N[2], thr = fluid_threads(h, 0, L, grid, 0);
  const size_t sm = spectrum_pass_smem(h.plan[0], L);
  const FastDiv dL = make_fastdiv((unsigned)L), dn1 = make_fastdiv((unsigned)h.n1);
  by_gaps(h.plan[0], [&](auto g) {
    constexpr bool G = decltype(g)::value;
    if (fwd && change) kwb_launch(k_eos_x_fwd<G, true>, grid, thr, sm, st, h, dL, dn1, step_s);
    else if (fwd) kwb_launch(k_eos_x_fwd<G, false>, grid, thr, sm, st, h, dL, dn1, step_s);
    else kwb_launch(k_eos_x_inv<G>, grid, thr, sm, st, h, dL, dn1, step_s, h.ndim == 1 ? 1 : 0);
  });
  return cudaGetLastError();
}
cudaError_t generic_spec(const SimDev &h, int axis, int op, long long step_s, cudaStream_t st) {
  const int L = h.L_spec[axis], grid = cdiv(h.n1, L) * (axis == 1 ? h.N[2] : h.N[1]);
  by_gaps(h.plan[axis], [&](auto g) {
    kwb_launch(k_spec_pass<decltype(g)::value>, grid, fluid_threads(h, axis, L, grid, 0),
               spectrum_pass_smem(h.plan[axis], L), st, h, axis, op, make_fastdiv((unsigned)L), step_s);
  });
  return cudaGetLastError();
}
// A gradient pass along an axis: CTAs, threads, shared memory, and whether a thread has 12 elements or
// more of a field (k_el_grad's U).  Long lines of a grid that gives each SM one CTA or two ask for so much
// shared memory that no SM takes more: launched while the kernel before still runs, they went two and
// three to the SMs that came free first (4096 x 256, 128 CTAs: 157 -> 109 us a step).
struct ElPass {
  int grid, thr;
  bool deep;
  size_t smem;
};
ElPass el_pass(const SimDev &h, int axis) {
  const FftPlan &pl = h.plan[axis];
  const int L = h.L_line[axis];
  ElPass p;
  p.grid = axis == 0 ? cdiv(h.N[1], 2 * L) * h.N[2] : cdiv(h.N[0], 2 * L) * (axis == 1 ? h.N[2] : h.N[1]);
  p.thr = pass_threads(pl, L, h.thr_line[axis]);
  p.deep = L * pl.n / p.thr >= 12;
  p.smem = line_pass_smem(pl, L);
  const int each = cdiv(p.grid, h.num_sms);
  if (p.deep && each <= 2) p.smem = std::max(p.smem, (size_t)228 * 1024 / (each + 1));
  return p;
}
// op with the kernel of such a pass
template <class Op>
auto by_el_kernel(const FftPlan &pl, int axis, bool deep, Op &&op) {
  return by_gaps(pl, [&](auto g) {
    constexpr bool G = decltype(g)::value;
    if (axis == 0) return deep ? op(k_el_grad<true, G, 8>) : op(k_el_grad<true, G, UNROLL>);
    return deep ? op(k_el_grad<false, G, 8>) : op(k_el_grad<false, G, UNROLL>);
  });
}
cudaError_t generic_el_prime(const SimDev &h) {
  cudaError_t e = cudaSuccess;
  for (int a = 0; a < h.ndim && e == cudaSuccess; ++a) {
    const ElPass p = el_pass(h, a);
    e = by_el_kernel(h.plan[a], a, p.deep, [&](auto k) { return raise_dynamic_smem((const void *)k, p.smem); });
  }
  return e;
}
cudaError_t generic_el_grad(const SimDev &h, int axis, const ElGrad &g, long long s, cudaStream_t st) {
  const ElPass p = el_pass(h, axis);
  by_el_kernel(h.plan[axis], axis, p.deep, [&](auto k) {
    kwb_launch(k, p.grid, p.thr, p.smem, st, h, axis, g, make_fastdiv((unsigned)h.L_line[axis]), s);
    return cudaSuccess;
  });
  return cudaGetLastError();
}
// Every length that fits: one launch against the passes, us a step, 16 points 4.7 / 20.7, 64 5.7 / 14.4, 512
// 9.4 / 18.2, 1024 13.7 / 26, 2048 25 / 44, 4096 44 / 71 (the passes with a measured schedule).
bool steps1d_fits(const SimDev &h) {
  return h.ndim == 1 && !h.elastic && h.plan[0].m == 0 && steps1d_smem(h) <= 200 * 1024;
}
cudaError_t steps1d_prime(const SimDev &h) {
  return by_gaps(h.plan[0], [&](auto g) { return raise_dynamic_smem((const void *)k_steps_1d<decltype(g)::value>, steps1d_smem(h)); });
}
cudaError_t build_eos1d(float2 *out, const float *M, int N, cudaStream_t st) {
  k_eos1d<<<cdiv(N, 256), 256, 0, st>>>(out, M, N);
  return cudaGetLastError();
}
cudaError_t launch_steps1d(const SimDev &h, const Groups1D &g, long long t_first, int steps, cudaStream_t st) {
  by_gaps(h.plan[0], [&](auto gaps) {
    k_steps_1d<decltype(gaps)::value><<<1, std::max(32, std::min(KWB_PASS_THREADS_MAX, (h.N[0] + 31) / 32 * 32)), steps1d_smem(h), st>>>(
        h, g, t_first, steps);
  });
  return cudaGetLastError();
}

}  // namespace kwb
