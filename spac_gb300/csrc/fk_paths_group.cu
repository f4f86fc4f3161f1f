// Time-parallel path kernel: a group of G lanes per path, G steps at a time.
//
// Where sigma, the drift and the potential are constant (every problem of the
// reference: Franke, both Monegros variants, and the disk problem), a path's
// positions are a running sum of normals that are known from the step's
// counter alone.  The lanes of a group form G steps' normals at once, a scan
// gives the G positions, every lane evaluates the source and the exit test at
// its own step, and the first step that stops ends the path.  The sums are those
// of one lane stepping G times, in another order: a round's normals are added
// in 2^-55 units (an error of 2^-56 each, times sigma sqrt(h), below the last
// digit of a position of order 1), and the source terms by lane.
//
// What bounds it: in the lane-per-path kernel a call cannot end before its
// longest path has run step by step, 1.4 us each for a warp on its own, while
// most lanes have nothing left to do (1,000 paths from one point: 0.48 ms; the
// circle mesh of the serial driver at h = 1e-5, whose longest path has 19,000
// steps: 17.5 ms).  Here a path of n steps takes n / G rounds; the price is
// the rest of the last round, G / 2 steps a path on average.  group_width()
// weighs the two.
//
// FP64 stepping only: FP32 positions would round differently summed in
// another order.  Point solves and arc stencils (the reference's meshes).
#include "fk_paths_kernel.cuh"

namespace fk {

namespace {

// Y of the paths after each step is Y0 (1 + c h)^n (Euler, constant c).
template <int PROB, int ST, bool CV, int G>
__global__ void __launch_bounds__(256, 2) paths_group_kernel(const LaunchArgs a) {
  using R = double;
  constexpr int NG = 32 / G;  // groups (paths) per warp
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ ExitQueue<R, false> sq[kMaxBlockWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gl = lane % G;                                                      // step of the round
  const unsigned gmask = G == 32 ? kFull : ((1u << G) - 1u) << (lane - gl);    // the group's lanes
  const size_t nodes_bytes = paths_slot_bytes(0, ST, 0, a.smem_nodes);
  double* sth = reinterpret_cast<double*>(smem_raw + sizeof(fx::Tables) + warp * nodes_bytes);
  stage_tables(smem_raw);
  ExitQueue<R, false>& q = sq[warp];
  for (;;) {
    int c = 0;
    if (lane == 0) c = atomicAdd(a.queue, 1);
    c = __shfl_sync(kFull, c, 0);
    if (c >= a.n_chunks) break;
    const ChunkDev ch = a.chunks[c];
    const ItemDev& itg = a.items[ch.item];
    const unsigned n_ch = ch.p1 - ch.p0;
    ArcDev sarc;
    if (ST == 1) {
      sarc = a.arcs[itg.stencil];
      __syncwarp();
      for (int i = lane; i < sarc.n; i += 32) sth[i] = a.arc_theta[sarc.theta_off + i];
      __syncwarp();
    }
    BvpDev bvp = a.bvp[itg.bvp];
    bvp.tab = reinterpret_cast<const fx::Tables*>(smem_raw);
    const bool cv = CV && bvp.cv == 1;
    const R d0 = bvp.dom[0], d1 = bvp.dom[1], d2 = bvp.dom[2], d3 = bvp.dom[3];
    const R h = itg.h, sqrth = itg.sqrth, x0 = itg.x, y0 = itg.y;
    const R s0 = itg.sub[0], s1 = itg.sub[1], s2 = itg.sub[2], s3 = itg.sub[3];
    const bool has_sub = (ST != 0) || itg.sub_shape >= 0;
    const bool sub_circle = (ST == 1) || itg.sub_shape == 1;
    const bool dom_can_win = domain_can_win<PROB>(has_sub, sub_circle, d0, d1, d2, d3, s0, s1, s2, s3);
    const R sg = Problem<PROB>::template sigma_of<R>(R(0));
    const R sh = sg * sqrth;
    const ExitTest<R, PROB> test(dom_can_win, has_sub, sub_circle, d0, d1, d2, d3, s0, s1, s2, s3, R(kGobet) * sh);
    // (1 + c h)^gl and (1 + c h)^G
    StepCoef<R> co;
    R pw = R(1), pwG = R(1), pw1 = R(1);
    if constexpr (!TraitsOf<PROB>::no_potential) {
      pw1 = R(1) + Problem<PROB>::potential * h;
      for (int i = 0; i < G; ++i) {
        if (i == gl) pw = pwG;
        pwG *= pw1;
      }
    }
    AccD acc[kNumAcc];
    unsigned long long n_steps = 0;
    unsigned n_dom = 0, n_cap = 0, n_done = 0;
    unsigned pl = lane / G, wnext = NG;
    bool active = pl < n_ch;
    R xs = x0, ys = y0, Y = R(1), Z = R(0), xi = R(0);  // the round's start; the lane's part of Z and xi
    int k = 0;
    int qn = 0;
    for (;;) {
      const bool any = __any_sync(kFull, active);
      if (!any && qn == 0) break;
      if (any) {
        // ---- G Euler steps: step k + gl of the group's path in lane gl
        const int n = k + gl;
        const uint4 r = philox10_rk(make_uint4(static_cast<uint32_t>(n), ch.p0 + pl, static_cast<uint32_t>(ch.item), a.stream),
                                    a.rkey);
        // (the normals' running sums as integers, 2^-55 units: 32 normals stay below
        // 2^63, the sums are exact and off the FP64 pipe)
        fx::u64 m0, m1;
        fx::u32 n0, n1;
        int ez;
        fx::normal_parts(bvp.tab, r.x, r.y, m0, m1, n0, n1, ez);
        fx::i64 zx = fx::normal_fx<55>(m0, n0, ez), zy = fx::normal_fx<55>(m1, n1, ez);
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
          const fx::i64 ux = __shfl_up_sync(kFull, zx, o, G), uy = __shfl_up_sync(kFull, zy, o, G);
          if (gl >= o) {
            zx += ux;
            zy += uy;
          }
        }
        const R x = xs + sh * fx::to_double(zx, -55), y = ys + sh * fx::to_double(zy, -55);
        R xp = __shfl_up_sync(kFull, x, 1, G), yp = __shfl_up_sync(kFull, y, 1, G);  // the step's start point
        if (gl == 0) {
          xp = xs;
          yp = ys;
        }
        Problem<PROB>::step(bvp, xp, yp, R(0), sg, cv, co);
        const bool capped = n + 1 >= a.max_steps;
        const bool out = active && (capped || !test.inside(x, y));
        const unsigned om = __ballot_sync(kFull, out);
        const unsigned og = om & gmask;
        const int first = __ffs(og) - 1;  // the lane whose step stops the path, or -1
        if (active && (first < 0 || lane <= first)) {
          const R Yn = TraitsOf<PROB>::no_potential ? R(1) : Y * pw;
          Z += TraitsOf<PROB>::no_potential ? co.f * h : (co.f * Yn) * h;
          if (cv) {
            // (the normals with all their digits: the term is as exact as they are)
            const R F = co.Fx * (sqrth * fx::to_double(m0, n0, ez)) + co.Fy * (sqrth * fx::to_double(m1, n1, ez));
            xi += TraitsOf<PROB>::no_potential ? F : Yn * F;
          }
        }
        if (om) {
          // ---- paths that stop: their sums, exit points and places in the queue
          R zt = Z, xt = xi;
#pragma unroll
          for (int o = 1; o < G; o <<= 1) {
            zt += __shfl_xor_sync(kFull, zt, o);
            if (CV) xt += __shfl_xor_sync(kFull, xt, o);
          }
          const unsigned em = __ballot_sync(kFull, lane == first);
          const unsigned me = em & gmask;
          const int rank = me ? __popc(em & ((me & (0u - me)) - 1u)) : 0;
          if (lane == first) {
            const int e = qn + rank;
            q.x[e] = x; q.y[e] = y; q.Z[e] = zt;
            q.Y[e] = TraitsOf<PROB>::no_potential ? R(1) : Y * pw * pw1;
            if (CV) q.xi[e] = xt;
            q.kf[e] = static_cast<unsigned>(n + 1) | (capped ? 1u << 31 : 0u);
          }
          if (first >= 0) {
            pl = wnext + rank;
            active = pl < n_ch;
            xs = x0; ys = y0; Y = R(1); Z = R(0); xi = R(0);
            k = -G;
          }
          wnext += __popc(em);
          qn += __popc(em);
          __syncwarp();
        }
        const R xe = __shfl_sync(kFull, x, G - 1, G), ye = __shfl_sync(kFull, y, G - 1, G);
        if (first < 0) {
          xs = xe;
          ys = ye;
          Y *= pwG;
        }
        k += G;
      }
      if (qn >= 32 || (!any && qn > 0)) {
        // ---- the top queued exits, one per lane (Reduce_Analytic, FeynmanKacSolver.cpp:198-292)
        const int cnt = qn < 32 ? qn : 32, qb = qn - cnt;
        R Yv = R(0), th = R(0);
        bool sub_exit = false;
        if (lane < cnt) {
          const int e = qb + lane;
          const R Zv = q.Z[e], xv = CV ? q.xi[e] : R(0);
          Yv = q.Y[e];
          const unsigned kf = q.kf[e];
          const bool cp = (kf >> 31) & 1u;
          Bnd<R> w;
          bool dw;
          dentro_exit<PROB>(q.x[e], q.y[e], dom_can_win, has_sub, sub_circle, d0, d1, d2, d3, s0, s1, s2, s3, w, dw);
          const R ex = w.ex, ey = w.ey;
          sub_exit = (ST != 0) && !dw;
          const R g = Problem<PROB>::u(bvp, ex, ey);
          const R score = Zv + Yv * g, vr = score + xv;
          acc[0].add(score);
          acc[1].add(score * score);
          if constexpr (CV) {
            acc[2].add(xv + xv * xv);
            acc[3].add(vr);
            acc[4].add(vr * vr);
            acc[5].add(xv * score);
            acc[7].add(xv * xv);
          }
          acc[6].add(sub_exit ? Zv + xv : vr);
          n_steps += kf & 0x3fffffffu;
          n_dom += dw ? 1u : 0u;
          n_cap += cp ? 1u : 0u;
          ++n_done;
          if (ST == 1 && sub_exit) th = arc_theta(sarc.interior, ex - sarc.cx, ey - sarc.cy);
        }
        if (ST == 1) {
          // Interfaz::Update_G moments, lanes over the arc's nodes
          const unsigned sm = __ballot_sync(kFull, sub_exit);
          if (sm) add_arc_moments(a.acc + itg.acc_off, sm, th, Yv, sth, sarc.n, sarc.c2, lane);
        }
        qn = qb;
        __syncwarp();
      }
    }
    add_item_sums<CV>(a, ch.item, acc, n_steps, n_dom, n_cap, n_done, lane);
  }
}

template <int PROB, int G>
const void* group_fn_p(int st, bool cv) {
  if (st == 1)
    return cv ? reinterpret_cast<const void*>(&paths_group_kernel<PROB, 1, true, G>)
              : reinterpret_cast<const void*>(&paths_group_kernel<PROB, 1, false, G>);
  return cv ? reinterpret_cast<const void*>(&paths_group_kernel<PROB, 0, true, G>)
            : reinterpret_cast<const void*>(&paths_group_kernel<PROB, 0, false, G>);
}
const void* group_fn(int problem, int st, bool cv, int g) {
  const void* fn = nullptr;
  with_problem(problem, [&](auto t) {
    constexpr int P = decltype(t)::value;
    if constexpr (TraitsOf<P>::const_sigma && TraitsOf<P>::no_drift)
      fn = g == 32 ? group_fn_p<P, 32>(st, cv) : group_fn_p<P, 8>(st, cv);
    return 0;
  });
  return fn;
}

}  // namespace

bool paths_group_available(int problem, int precision, int stencil_kind) {
  return precision == 0 && stencil_kind <= 1 && group_fn(problem, stencil_kind, false, 32) != nullptr;
}

cudaError_t launch_paths_group(const LaunchArgs& a, int problem, int g, int grid, int block, cudaStream_t s) {
  const void* fn = group_fn(problem, a.stencil_kind, a.any_cv != 0, g);
  if (!fn || block < 32 || block > 256 || block % 32 != 0) return cudaErrorInvalidValue;
  const size_t smem = sizeof(fx::Tables) + (block / 32) * paths_slot_bytes(0, a.stencil_kind, 0, a.smem_nodes);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<LaunchArgs*>(&a)};
  return cudaLaunchKernel(fn, dim3(grid), dim3(block), args, smem, s);
}

}  // namespace fk
