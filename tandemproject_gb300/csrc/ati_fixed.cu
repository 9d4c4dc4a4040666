// ati_fixed.cu — 64-bit fixed-point line sweeps of the FP64 fast path (see ati_fixed.h).
//
// k_sweep_fix is the segmented line solve of k_sweep_seg (ati_kernels.cu) in integers: 32 consecutive lines of one
// block and one field staged whole in shared memory as a [point][line] tile, one warp per segment of about 48 points,
// lane l line l, segment carries handed on by one warp (src/Subroutines3D.f90:84-206).
//
// The solve itself, its scales and its errors: ati_fixed_line.h.
//
// Bound: integer issue and the latency of its chains.  A row takes some 230 warp instructions, 33 of them 64-bit
// multiply-adds of 4 clocks, at 15 warps an SM (128 registers a thread; the tiles fill the shared memory): half of the
// issue slots, the FP64 pipe a sixth busy with the conversions out, DRAM at 20-25 %.  Clocks a row of a warp, of some 1700
// along eta: staging 150, scales and conversions 320, elimination 570, back substitution 320, results 390.  On 8.85 M
// points (4.5 fields a launch, 2070 MHz): xi 795 -> 500 us, eta 754 -> 486, zeta 764 -> 407 a derivative launch, the xi and
// eta filters 1093 -> 583 and 954 -> 625, against the FP64 sweeps (k_sweep_xc, k_sweep_g), which keep the FP64 pipe
// 86-91 % busy.  (With one scale for a whole line: xi 450, eta 384, zeta 385, but rows well below the line's largest lost
// accuracy.)
#include <cuda_runtime.h>

#include <cstdint>

#include "ati_fixed.h"
#include "ati_fixed_line.h"

namespace ati {
namespace fast {
namespace {

template <int NN>
__device__ __forceinline__ bool line_of(const BlockDev &B, int t, int64_t &base, int64_t &stride, int &jk) {
  const int nx = B.lxi + 1, ny = B.let + 1, nz = B.lze + 1;
  if (NN == 1) {
    base = B.off + (int64_t)t * nx; stride = 1; jk = t;
    return t < ny * nz;
  } else if (NN == 2) {
    const int xi = t % nx, ze = t / nx;
    base = B.off + (int64_t)ze * nx * ny + xi; stride = nx; jk = xi * nz + ze;
    return t < nx * nz;
  }
  base = B.off + t; stride = (int64_t)nx * ny; jk = t;
  return t < nx * ny;
}

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

constexpr int RS = SEG_LINES + 1;  // tile row stride in doubles: rows and columns of a tile are free of bank conflicts

// (128 registers a thread: xi, eta and zeta derivatives of 8.85 M points took 487, 472, 387 us at 128, 497, 502, 433 at 112,
// where it spills, 706, 478, 416 at 168, where fewer CTAs fit)
template <int NN, bool FILT>
__global__ void __maxnreg__(128) k_sweep_fix(const __grid_constant__ FixArgs a) {
  extern __shared__ __align__(16) unsigned char fx_smem[];
  const int nwarp = (int)(blockDim.x >> 5);
  const LTile LT = a.lt[blockIdx.x];
  const BlockDev &B = a.blk[LT.b];
  const int f = blockIdx.y;
  const int lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5);
  const int L = NN == 1 ? B.lxi + 1 : (NN == 2 ? B.let + 1 : B.lze + 1);
  const int t0 = LT.t0, nx = B.lxi + 1;
  const int nl = t0 >= B.nbsize[NN] ? 0
                 : (NN == 2 && a.rowtiles) ? min(SEG_LINES, nx - t0 % nx)
                                           : min(SEG_LINES, (int)B.nbsize[NN] - t0);
  // shared memory: per segment and line the two values passed on and received, their scales (before them the exponent
  // maxima), then the tile
  longlong2 *cf = reinterpret_cast<longlong2 *>(fx_smem), *cx = cf + nwarp * SEG_LINES;
  unsigned *smax = reinterpret_cast<unsigned *>(cx + nwarp * SEG_LINES);
  short2 *sw = reinterpret_cast<short2 *>(smax);
  double *tile = reinterpret_cast<double *>(smax + nwarp * SEG_LINES);
  int64_t base = 0, stride = 1;
  int jk = 0;
  line_of<NN>(B, t0 + lane, base, stride, jk);
  const double *in = a.io.in + f * a.io.in_fs;

  // 1. stage the lines
  if constexpr (NN == 1) {
    const double *src0 = in + B.off + (int64_t)t0 * L;
    for (int ln = w; ln < nl; ln += nwarp) {
      const double *src = src0 + (int64_t)ln * L + lane;
      double *dst = tile + lane * RS + ln;
#pragma unroll 4
      for (int i = lane; i < L; i += 32, src += 32, dst += 32 * RS) cp_async8(dst, src);
    }
  } else {
    if (lane < nl) {
      const double *src = in + base + (int64_t)w * stride;
      const int64_t step = (int64_t)nwarp * stride;
      double *dst = tile + w * RS + lane;
#pragma unroll 4
      for (int i = w; i < L; i += nwarp, src += step, dst += nwarp * RS) cp_async8(dst, src);
    }
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();

  const int S = seg_count(L);
  const bool act = w < S && lane < nl, multi = S > 1;
  double *col = tile + lane;
  const int *rows = a.rows + (int64_t)B.fac_off[NN] * FX_RT;
  const int *et = reinterpret_cast<const int *>(a.ends + ((int64_t)LT.b * 3 + NN - 1) * FX_ET);
  const bool per = !FILT && NN == 3 && B.ndf[0][NN] == 1;  // both faces periodic onto this block
  fxl::Segment<FILT, !FILT && NN == 3, RS> sg(rows, et, col, L, S, w, per, a.fs);
  const int me = w * SEG_LINES + lane;
  auto put_pair = [&](longlong2 *c, int at, const fxl::Pair &p) { c[at] = make_longlong2(p.a, p.b); };
  auto pair = [&](const longlong2 *c, int at, int W) { return fxl::Pair{c[at].x, c[at].y, W}; };

  // 2. scales and integers
  if (act) smax[me] = sg.maxima();
  __syncthreads();
  if (act) {
    unsigned mx = 0;
    for (int k = 0; k < S; k++) mx = max(mx, smax[k * SEG_LINES + lane]);
    sg.convert(mx);
    cf[me] = make_longlong2((long long)sg.sc.M, (long long)sg.sc.edge);
  }
  __syncthreads();
  if (act)
    sg.reads([&](int k) {
      const longlong2 v = cf[k * SEG_LINES + lane];
      return fxl::Scales{(fxl::u64)v.x, (fxl::u64)v.y};
    });
  __syncthreads();

  // 3. the segments' forward eliminations, and the values carried from one to the next by the first warp
  fxl::Pair c{0, 0, fxl::NONE}, x = c, y = c;
  if (act) {
    c = sg.forward();
    if (multi) {
      put_pair(cf, me, c);
      sw[me].x = (short)c.W;
    }
  }
  if (multi) {
    __syncthreads();
    if (w == 0 && lane < nl) {
      fxl::Pair v{0, 0, fxl::NONE};
      for (int k = 1; k < S; k++) {
        const int at = (k - 1) * SEG_LINES + lane;
        v = fxl::carry_forward(rows, seg_start(k, L, S), pair(cf, at, sw[at].x), v);
        put_pair(cx, at + SEG_LINES, v);
        sw[at + SEG_LINES].y = (short)v.W;
      }
    }
    __syncthreads();
  }
  double *out = a.io.out + f * a.io.out_fs;
  double *out2 = FILT && a.io.out2 ? a.io.out2 + f * a.io.out_fs : nullptr;
  const bool odd = sg.bad || sg.pre != 0;
  constexpr bool DIRECT = NN != 1 && !FILT;  // one-segment lines write their results from the back substitution
  // 4. back substitutions; one-segment derivatives along eta and zeta go straight to DRAM from there
  if (act) {
    if (DIRECT && !multi && !odd) {
      double *po = out + base + (int64_t)(L - 1) * stride;
      sg.backward([&](int, fxl::i64 q, int W) {
        *po = fxl::from_fixed(q, sg.out(W) * (1 << 20));
        po -= stride;
      });
    } else {
      c = sg.backward([&](int i, fxl::i64 q, int) { sg.set(i, q); });
      if (multi) {
        if (w > 0) x = pair(cx, me, sw[me].y);
        c = sg.with_incoming(c, x);
        put_pair(cf, me, c);
        sw[me].x = (short)c.W;
      }
    }
  }
  if (multi) {
    __syncthreads();
    if (w == 0 && lane < nl) {
      fxl::Pair v{0, 0, fxl::NONE};
      for (int k = S - 2; k >= 0; k--) {
        const int at = (k + 1) * SEG_LINES + lane;
        v = fxl::carry_backward(rows, seg_start(k + 1, L, S), pair(cf, at, sw[at].x), v);
        put_pair(cx, at - SEG_LINES, v);
        sw[at - SEG_LINES].y = (short)v.W;
      }
    }
    __syncthreads();
  }
  // 5. results: eta/zeta rows straight to DRAM, xi lines through the tile
  if (act) {
    if (multi || !DIRECT || odd) {
      if (multi && w < S - 1) y = pair(cx, me, sw[me].y);
      double *po = out + base + (int64_t)sg.s0 * stride;
      auto put = [&](int i, double r) {
        if constexpr (NN == 1) {
          col[i * RS] = r;
        } else {
          if (FILT) {  // rr = rr + sb (src/Subroutines3D.f90:200-202)
            r = in[po - out] + r;
            if (out2) out2[po - out] = r;
          }
          *po = r;
          po += stride;
        }
      };
      if (odd)
        sg.results(x, y, [&](int i, fxl::i64 v, int W) {
          put(i, sg.bad ? __hiloint2double(0x7ff80000, 0) : ldexp((double)v, sg.out(W)));
        });
      else
        sg.results(x, y, [&](int i, fxl::i64 v, int W) { put(i, fxl::from_fixed(v, sg.out(W) * (1 << 20))); });
    }
    if (!FILT && a.io.drva) {  // the line ends, read back from this thread's own stores
      double *drv = a.drva + B.face_off[NN] * 10 + jk + (int64_t)B.nbsize[NN] * (a.io.m0 + f - 1);
      const double *r = NN == 1 ? col : out + base;
      const int64_t rs = NN == 1 ? RS : stride;
      if (w == 0) drv[0] = r[0];                                                     // drva(jk,m,0) = sb(is)
      if (w == S - 1) drv[(int64_t)B.nbsize[NN] * 5] = r[(L - 1) * rs];  // drva(jk,m,1) = sb(ie)
    }
  }
  if constexpr (NN == 1) {
    __syncthreads();
    const int64_t o0 = B.off + (int64_t)t0 * L;
    auto wr = [&](int64_t p, double v, double q) {
      const double r = FILT ? q + v : v;  // rr = rr + sb (src/Subroutines3D.f90:200-202)
      out[p] = r;
      if (out2) out2[p] = r;
    };
    for (int ln = w; ln < nl; ln += nwarp) {
      const int64_t lb = o0 + (int64_t)ln * L;
      int i = lane;
      for (; i + 96 < L; i += 128) {  // the filter runs in place: four inputs read before any is stored
        double q0 = 0, q1 = 0, q2 = 0, q3 = 0;
        if (FILT) { q0 = in[lb + i]; q1 = in[lb + i + 32]; q2 = in[lb + i + 64]; q3 = in[lb + i + 96]; }
        wr(lb + i, tile[i * RS + ln], q0);
        wr(lb + i + 32, tile[(i + 32) * RS + ln], q1);
        wr(lb + i + 64, tile[(i + 64) * RS + ln], q2);
        wr(lb + i + 96, tile[(i + 96) * RS + ln], q3);
      }
      for (; i < L; i += 32) wr(lb + i, tile[i * RS + ln], FILT ? in[lb + i] : 0.0);
    }
  }
}

size_t fixed_smem(int nwarp, int maxlen) {
  return (size_t)nwarp * SEG_LINES * (2 * sizeof(longlong2) + sizeof(unsigned)) + (size_t)maxlen * RS * sizeof(double);
}

template <typename K>
cudaError_t max_smem(K kernel) {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa{};
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
}

}  // namespace

cudaError_t fixed_init() {
  cudaError_t e = max_smem(k_sweep_fix<1, false>);
  if (e == cudaSuccess) e = max_smem(k_sweep_fix<2, false>);
  if (e == cudaSuccess) e = max_smem(k_sweep_fix<3, false>);
  if (e == cudaSuccess) e = max_smem(k_sweep_fix<1, true>);
  if (e == cudaSuccess) e = max_smem(k_sweep_fix<2, true>);
  return e;
}

void sweep_fixed(const Eng<double> &e, cudaStream_t st, int nn, bool filt, const SweepIO<double, double> &io) {
  FixArgs a;
  a.blk = e.blk;
  a.rows = e.fxr[filt];
  a.ends = e.fxe[filt];
  a.io = io;
  a.drva = e.drva;
  a.fs = e.fx_scale[filt];
  a.rowtiles = e.eta_rowtiles;
  for (int c = 0; c < e.nsegc[nn]; c++) {  // one launch per class of equal segment counts
    const SegClass &C = e.segc[nn][c];
    if (C.n == 0) continue;
    a.lt = e.lts[nn] + C.off;
    const int nt = SEG_LINES * seg_count(C.maxlen);
    const size_t smem = fixed_smem(seg_count(C.maxlen), C.maxlen);
    const dim3 g(C.n, io.nf);
    // The directions' and classes' sweeps of a stage run at once, and an SM runs kernels side by side only at one split
    // of its memory between L1 and shared memory: on a small handle, whose sweeps together fit the GPU, each asks for
    // the largest share, so that none waits for an SM to drain (a step of 0.23 M points 1170 -> 967 us; of 0.6 to 1.9 M
    // the same; of 3.5 M, where each sweep fills the GPU and the tables want the L1, 8139 -> 8230 us).
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = g;
    cfg.blockDim = nt;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = e.N < (1 << 20) ? 1 : 0;
    auto launch = [&](auto *k) { (void)cudaLaunchKernelEx(&cfg, k, a); };
    if (!filt) {
      if (nn == 1) launch(k_sweep_fix<1, false>);
      else if (nn == 2) launch(k_sweep_fix<2, false>);
      else launch(k_sweep_fix<3, false>);
    } else {
      if (nn == 1) launch(k_sweep_fix<1, true>);
      else launch(k_sweep_fix<2, true>);
    }
  }
}

}  // namespace fast
}  // namespace ati
