// Two-pass NTT / INTT kernels for sm_100a that meet in the L2 cache.
//
// A limb is a 256 x 256 matrix (row-major). The forward transform runs the
// eight stages that pair rows in a column pass (one CTA per tile of 16
// columns: 64-byte row segments, transposition through shared memory) and the
// eight stages inside rows in a row pass (one warp per two rows, exchange with
// __syncwarp only). The inverse transform is the mirror image. Both passes are
// plain grids of independent 128-thread CTAs: no cluster, no cross-CTA wait.
//
// What keeps two passes near one trip to HBM: the second pass works in place on
// what the first just wrote, and up to about 400 limbs (100 MiB) that is still
// in the 126 MB L2. Chunks of kChunkJobs limbs per launch pair: the passes are
// bound by instruction issue, and the ramp and tail of more launches cost more
// than the second trip saves (640 limbs there and back: 341 us in chunks of
// 192, 334 in 320, 320 in one).
// These kernels take calls of every size. Kernels that streamed tiles with bulk
// tensor copies and kept a prime's twiddles in shared memory, once used from
// 256 limb transforms on, took 15 to 19 % longer forwards and within 2 % the
// same time backwards, but for 8 x 59 limbs, where they took 3 % less (us, both
// timed in turn, calls queued up; forward and inverse of the removed | of these):
// 8 x 32 limbs 71.6 66.9 | 61.1 66.0, 8 x 59 123.2 115.5 | 107.3 118.9, 12 x 40
// 123.0 114.5 | 106.9 115.9, 16 x 40 160.6 151.3 | 139.1 150.3, 32 x 47 385 361 |
// 328 358. Repeated for more than 0.2 s both run into the power limit (1000 W; 1765
// MHz | 1610 MHz), which leaves 337 | 333 us for 16 x 40 there and back.
//
// The per-thread arithmetic (radix-16 register phases, Shoup twiddles, lazy
// [0,4q) butterflies for primes below 2^30) is shared with the cluster
// kernels (ntt_core.cuh); the two implementations produce the same words.
#include "context.h"

namespace cfhe {
namespace {

constexpr int kTpThreads = 128;
constexpr int kColTile = 16;   // columns per CTA in the column pass
constexpr int kChunkJobs = 640;
// CTAs an SM holds (80 and 64 registers a thread). Measured on 188 limbs:
// 6 and 8 are the best of 5 to 10 each, or within 2 % of it.
constexpr int kColCtas = 6, kRowCtas = 8;
// column-pass buffer: word (r, x) at r*16 + x + 16*(r >> 4): both the
// (r0 + 16k) and the (16g + k) access of a half-warp are 128 contiguous bytes
// on banks of their own
constexpr int kColBufWords = 256 * kColTile + 256;
// row-pass buffer of a warp: two rows, 272 words apart so that the strided
// accesses of the two half-warps fall on different banks; inside a row the
// 16-byte chunks of every block of 16 words are permuted by the block number,
// so that the block accesses (128 bits a lane, 64 bytes between lanes) do too
constexpr int kRowPitch = 272;
constexpr int kRowBufWordsCta = kTpThreads / 32 * 2 * kRowPitch;

struct Job {
  int p, l;
  uint32_t q;
  const Tw *tw;
  const uint4 *row_tw;
  const uint32_t *src;
  uint32_t *dst;
};

__device__ __forceinline__ Job get_job(const NttArgs &a, const uint4 *row_table, int t) {
  Job j;
  j.p = t / a.n_limbs;
  j.l = t - j.p * a.n_limbs;
  j.q = a.q[j.l];
  j.tw = a.table + (size_t)a.g[j.l] * kN;
  j.row_tw = row_table + (size_t)a.g[j.l] * (kN / 2);
  j.src = a.src + (size_t)j.p * a.src_poly_stride + (size_t)a.src_limb[j.l] * kN;
  j.dst = a.dst + (size_t)j.p * a.dst_poly_stride + (size_t)a.dst_limb[j.l] * kN;
  return j;
}

__device__ __forceinline__ int col_word(int r, int x) { return r * kColTile + x + 16 * (r >> 4); }

// twiddles of the in-row phase that works on blocks, thread g of row R: eight
// 16-byte chunks, each contiguous over the threads of the row
__device__ __forceinline__ void ld_row_tw(const uint4 *t, Tw *out) {
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const uint4 w = __ldg(t + c * 16);
    out[2 * c] = Tw{w.x, w.y};
    if (c < 7) out[2 * c + 1] = Tw{w.z, w.w};
  }
}

// Column passes: thread (x, hi) of 128 works on the two adjacent columns 2x,
// 2x + 1 of the tile, so that a fetched twiddle serves two butterflies and every
// access to memory moves 64 bits. (One column a thread: the 16 broadcast loads
// of twiddles per 16 words kept the load pipe as busy as the butterflies keep
// the multiplier; 62 cycles a word and warp against 54.)
// NARROW: word by word, for a forward source or an inverse destination that
// lies at an odd word (launch_ntt).
template <bool NARROW = false>
__device__ __forceinline__ void put2(uint32_t *p, uint32_t a, uint32_t b) {
  if constexpr (NARROW) {
    p[0] = a;
    p[1] = b;
  } else {
    *reinterpret_cast<uint2 *>(p) = make_uint2(a, b);
  }
}
template <bool NARROW = false>
__device__ __forceinline__ void get2(const uint32_t *p, uint32_t &a, uint32_t &b) {
  if constexpr (NARROW) {
    a = p[0];
    b = p[1];
  } else {
    const uint2 w = *reinterpret_cast<const uint2 *>(p);
    a = w.x;
    b = w.y;
  }
}

// ---- forward, pass 1: stages 1-8 (rows paired), src -> dst, values lazy ----
template <bool FAST, bool LATE, bool NARROW>
__device__ __forceinline__ void fwd_cols(const NttArgs &a, const Job &j, int tile, int tid,
                                         uint32_t *xbuf) {
  const uint32_t q = j.q, q2 = 2 * q;
  const int x = 2 * (tid & 7), hi = tid >> 3;
  uint32_t v[16], w[16];
  Tw t[15];
  const uint32_t *s = j.src + hi * kRowWords + kColTile * tile + x;
  ld_tw16(j.tw, 1, t);  // the tables are never written by a kernel: fetched before the wait
  pdl_wait();
#pragma unroll
  for (int k = 0; k < 16; k++) get2<NARROW>(s + k * 16 * kRowWords, v[k], w[k]);
  if (a.premul) {
    const Tw kc = a.kc[j.l];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      v[k] = shoup_mul(v[k], kc, q);
      w[k] = shoup_mul(w[k], kc, q);
    }
  }
  ct_radix16_pre<FAST>(v, t, q, q2);
  if constexpr (LATE) pdl_launch_dependents();
  ct_radix16_pre<FAST>(w, t, q, q2);
  ld_tw16(j.tw, 16 + hi, t);  // in flight across the transposition
#pragma unroll
  for (int k = 0; k < 16; k++) put2(xbuf + col_word(hi + 16 * k, x), v[k], w[k]);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 16; k++) get2(xbuf + col_word(16 * hi + k, x), v[k], w[k]);
  ct_radix16_pre<FAST>(v, t, q, q2);
  ct_radix16_pre<FAST>(w, t, q, q2);
  uint32_t *o = j.dst + (16 * hi) * kRowWords + kColTile * tile + x;
#pragma unroll
  for (int k = 0; k < 16; k++) put2(o + k * kRowWords, v[k], w[k]);
}

// ---- inverse, pass 2: strides 1..128 rows, per-limb constant, in place ----
template <bool FAST, bool LATE, bool NARROW>
__device__ __forceinline__ void inv_cols(const NttArgs &a, const Job &j, int tile, int tid,
                                         uint32_t *xbuf) {
  const uint32_t q = j.q, q2 = 2 * q;
  const int x = 2 * (tid & 7), hi = tid >> 3;
  uint32_t v[16], w[16];
  uint32_t *base = j.dst + kColTile * tile + x;
  Tw t[15];
  ld_tw16(j.tw, 16 + hi, t);
  pdl_wait();
#pragma unroll
  for (int k = 0; k < 16; k++) get2<NARROW>(base + (16 * hi + k) * kRowWords, v[k], w[k]);
  gs_radix16_pre<FAST>(v, t, q, q2);
  if constexpr (LATE) pdl_launch_dependents();
  gs_radix16_pre<FAST>(w, t, q, q2);
  ld_tw16(j.tw, 1, t);  // in flight across the transposition
#pragma unroll
  for (int k = 0; k < 16; k++) put2(xbuf + col_word(16 * hi + k, x), v[k], w[k]);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 16; k++) get2(xbuf + col_word(hi + 16 * k, x), v[k], w[k]);
  const Tw kc = a.kc[j.l], kcw = a.kcw[j.l];
  gs_radix16_last<FAST>(v, t, kc, kcw, q, q2);
  gs_radix16_last<FAST>(w, t, kc, kcw, q, q2);
  const uint32_t half = q >> 1;
  const bool centred = a.centred != 0;
  auto finish = [&](uint32_t r) {
    r = umin32(r, r - q);
    if (centred && r > half) r -= q;
    return r;
  };
#pragma unroll
  for (int k = 0; k < 16; k++) put2<NARROW>(base + (hi + 16 * k) * kRowWords, finish(v[k]), finish(w[k]));
}

// A warp owns two rows and exchanges through its own piece of shared memory: no
// barrier wider than the warp. Offsets of thread (row half, g):
struct RowPos {
  int strided[4];  // word g of block k: 16 k + strided[(k >> 1) & 3]
  int block[4];    // chunk c of block g
  __device__ __forceinline__ explicit RowPos(int lane) {
    const int base = (lane >> 4) * kRowPitch, g = lane & 15;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      strided[i] = base + 4 * ((g >> 2) ^ i) + (g & 3);
      block[i] = base + 16 * g + 4 * (i ^ ((g >> 1) & 3));
    }
  }
  // 128-bit word u (0..127) of the two rows, read or written in memory order
  static __device__ __forceinline__ int linear(int u) {
    const int k = (u & 63) >> 2;
    return (u >> 6) * kRowPitch + 16 * k + 4 * ((u & 3) ^ ((k >> 1) & 3));
  }
};

__device__ __forceinline__ void sts4(uint32_t *p, const uint32_t *v) {
  *reinterpret_cast<uint4 *>(p) = make_uint4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void lds4(const uint32_t *p, uint32_t *v) {
  const uint4 w = *reinterpret_cast<const uint4 *>(p);
  v[0] = w.x;
  v[1] = w.y;
  v[2] = w.z;
  v[3] = w.w;
}

// ---- forward, pass 2: stages 9-16 (inside rows), in place on dst ----
// The last phase leaves a thread 16 consecutive words. They go back through
// shared memory so that global memory sees whole lines: stored as they are
// (128 bits a lane, 64 bytes between lanes) the pass took 72 cycles a word and
// warp, this way 56.
template <bool FAST, bool LATE>
__device__ __forceinline__ void fwd_rows(const NttArgs &a, const Job &j, int pair, int lane, const RowPos &pos,
                                         uint32_t *buf) {
  const uint32_t q = j.q, q2 = 2 * q;
  const int g = lane & 15, R = 2 * pair + (lane >> 4);
  uint32_t v[16];
  Tw t[15];
  ld_tw16(j.tw, 256 + R, t);
  pdl_wait();
  const uint32_t *s = j.dst + R * kRowWords + g;
#pragma unroll
  for (int k = 0; k < 16; k++) v[k] = s[16 * k];
  ct_radix16_pre<FAST>(v, t, q, q2);
  if constexpr (LATE) pdl_launch_dependents();
  ld_row_tw(j.row_tw + R * 128 + g, t);  // in flight across the exchange
#pragma unroll
  for (int k = 0; k < 16; k++) buf[pos.strided[(k >> 1) & 3] + 16 * k] = v[k];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; i++) lds4(buf + pos.block[i], v + 4 * i);
  ct_radix16_pre<FAST>(v, t, q, q2);
  if (!a.ep_mode) {
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = ct_fold<FAST>(v[k], q, q2);
  }
#pragma unroll
  for (int i = 0; i < 4; i++) sts4(buf + pos.block[i], v + 4 * i);
  __syncwarp();
  uint4 *o = reinterpret_cast<uint4 *>(j.dst + 2 * pair * kRowWords);
  if (a.ep_mode) {
    // ModDown-family epilogue: (pad * x - ntt) * scale, canonical. The
    // transform's values enter as the last stage left them (below 4q, or 2q
    // for the large primes): a Shoup product takes any 32-bit word.
    const int l = j.l;
    const Tw scale = a.ep_scale[l], ps = a.ep_ps[l];
    const bool has_x = a.ep_limb[l] != 255, pad = a.ep_mode == 2;
    const uint4 *xp = reinterpret_cast<const uint4 *>(a.ep_src + (size_t)j.p * a.ep_poly_stride +
                                                      (size_t)(has_x ? a.ep_limb[l] : 0) * kN + 2 * pair * kRowWords);
    uint4 xv[4];
#pragma unroll
    for (int i = 0; i < 4; i++) xv[i] = has_x ? xp[lane + 32 * i] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      uint32_t y[4];
      lds4(buf + RowPos::linear(lane + 32 * i), y);
      const uint32_t x[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        if (pad) {
          // pad*scale*x - scale*ntt: two independent products
          uint32_t t1 = shoup_mul(x[e], ps, q), t2 = shoup_mul(y[e], scale, q);  // both below 2q
          if constexpr (FAST) {
            y[e] = ct_fold<true>(t1 - t2 + q2, q, q2);
          } else {
            t1 = umin32(t1, t1 - q);
            t2 = umin32(t2, t2 - q);
            const uint32_t r = t1 - t2 + q;  // (0, 2q)
            y[e] = umin32(r, r - q);
          }
        } else {
          uint32_t d;
          if constexpr (FAST)
            d = x[e] - umin32(y[e], y[e] - q2) + q2;  // (0, 3q)
          else
            d = x[e] - umin32(y[e], y[e] - q) + q;  // (0, 2q)
          d = shoup_mul(d, scale, q);
          y[e] = umin32(d, d - q);
        }
      }
      o[lane + 32 * i] = make_uint4(y[0], y[1], y[2], y[3]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) o[lane + 32 * i] = *reinterpret_cast<const uint4 *>(buf + RowPos::linear(lane + 32 * i));
  }
}

// ---- inverse, pass 1: strides 1..128 words (inside rows), src -> dst ----
template <bool FAST, bool LATE>
__device__ __forceinline__ void inv_rows(const NttArgs &, const Job &j, int pair, int lane, const RowPos &pos,
                                         uint32_t *buf) {
  const uint32_t q = j.q, q2 = 2 * q;
  const int g = lane & 15, R = 2 * pair + (lane >> 4);
  uint32_t v[16];
  Tw t[15];
  ld_row_tw(j.row_tw + R * 128 + g, t);
  pdl_wait();
  const uint4 *s = reinterpret_cast<const uint4 *>(j.src + 2 * pair * kRowWords);
  uint4 in[4];
#pragma unroll
  for (int i = 0; i < 4; i++) in[i] = s[lane + 32 * i];
#pragma unroll
  for (int i = 0; i < 4; i++) *reinterpret_cast<uint4 *>(buf + RowPos::linear(lane + 32 * i)) = in[i];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; i++) lds4(buf + pos.block[i], v + 4 * i);
  gs_radix16_pre<FAST>(v, t, q, q2);
  if constexpr (LATE) pdl_launch_dependents();
  ld_tw16(j.tw, 256 + R, t);  // in flight across the exchange
#pragma unroll
  for (int i = 0; i < 4; i++) sts4(buf + pos.block[i], v + 4 * i);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 16; k++) v[k] = buf[pos.strided[(k >> 1) & 3] + 16 * k];
  gs_radix16_pre<FAST>(v, t, q, q2);
  uint32_t *o = j.dst + R * kRowWords + g;
#pragma unroll
  for (int k = 0; k < 16; k++) o[16 * k] = v[k];
}

// Every pass fetches its first twiddles and waits for the kernel before it
// (pdl_wait). LATE: it lets the next kernel's CTAs in when its own words have
// arrived and gone through the first butterflies, otherwise at its top
// (launch_pass holds the rule).
// PASS 0: column pass, a CTA per tile; PASS 1: row pass, a warp per two rows.
// Forward runs 0 then 1; inverse 1 then 0. One tile per CTA: a grid that fills
// the GPU once and walks the tiles was 3 to 12 % slower (the SMs do not progress
// evenly, and a fixed share each leaves some of them waiting).
// Measured, 188 limbs of 47 primes in place: both passes 50.2 -> 40.8 us
// forward, 55.1 -> 45.7 us inverse (256-thread CTAs, one column a thread, row
// pass stored as the butterflies leave it); the butterflies alone take 28 us.
template <bool INV, int PASS, bool LATE, bool NARROW>
__global__ void __launch_bounds__(kTpThreads, PASS == 0 ? kColCtas : kRowCtas)
    ntt_twopass_kernel(const __grid_constant__ NttArgs a, const uint4 *row_table, int job0) {
  __shared__ __align__(16) uint32_t xbuf[PASS == 0 ? kColBufWords : kRowBufWordsCta];
  if constexpr (!LATE) pdl_launch_dependents();
  const int tid = threadIdx.x;
  if constexpr (PASS == 0) {
    constexpr int kTiles = kRowWords / kColTile;
    const Job j = get_job(a, row_table, job0 + blockIdx.x / kTiles);
    const int part = blockIdx.x % kTiles;
    const bool fast = j.q < (1u << 30);
    if constexpr (!INV) {
      if (fast) fwd_cols<true, LATE, NARROW>(a, j, part, tid, xbuf); else fwd_cols<false, LATE, NARROW>(a, j, part, tid, xbuf);
    } else {
      if (fast) inv_cols<true, LATE, NARROW>(a, j, part, tid, xbuf); else inv_cols<false, LATE, NARROW>(a, j, part, tid, xbuf);
    }
  } else {
    constexpr int kWarps = kTpThreads / 32, kCtas = kRowWords / 2 / kWarps;
    const int lane = tid & 31, warp = tid >> 5;
    uint32_t *buf = xbuf + warp * 2 * kRowPitch;
    const Job j = get_job(a, row_table, job0 + blockIdx.x / kCtas);
    const int pair = (blockIdx.x % kCtas) * kWarps + warp;
    const RowPos pos(lane);
    const bool fast = j.q < (1u << 30);
    if constexpr (!INV) {
      if (fast) fwd_rows<true, LATE>(a, j, pair, lane, pos, buf); else fwd_rows<false, LATE>(a, j, pair, lane, pos, buf);
    } else {
      if (fast) inv_rows<true, LATE>(a, j, pair, lane, pos, buf); else inv_rows<false, LATE>(a, j, pair, lane, pos, buf);
    }
  }
}

template <bool INV, int PASS>
cudaError_t launch_pass(const Context &ctx, const NttArgs &args, int job0, int cnt) {
  const int grid = PASS == 0 ? cnt * (kRowWords / kColTile) : cnt * (kRowWords / 2) / (kTpThreads / 32);
  // When the next kernel's CTAs are let in (GPU time, calls queued up, us):
  // * Late where the row pass fits the GPU at once (37 limbs). At the top, CTAs of
  //   several kernels ahead occupy the SMs while nothing of theirs can run, and
  //   small calls take as long as without early launches: 12 limbs 11.1 forward and
  //   12.2 inverse, late 7.4 and 8.1; 23 limbs 12.1 and 12.9, late 9.8 and 10.6;
  //   HMult at level 1 56.0, late 53.0, at level 7 75.0, late 71.9. (Right after
  //   the wait is as good up to 20 limbs, but 11.6 at 23.)
  // * At the top above that: the last CTAs start when the others are done, and
  //   every microsecond that they keep the next kernel out is lost: eight hoisted
  //   rotations at level 12 281.4, late 286.3, at level 28 607.6, late 613.0.
  // * Late again for inverse calls of more than 128 limbs (batches; the operators of
  //   the parameter sets have at most 112): 16 x 40 limbs 149.9, late 147.8, 32
  //   x 47 360.8, late 355.9; up to 3 x 47 both are within 1 %.
  const bool late = cnt * (kRowWords / 2) / (kTpThreads / 32) <= ctx.num_sms * kRowCtas || (INV && cnt > 128);
  auto kernel = late ? ntt_twopass_kernel<INV, PASS, true, false> : ntt_twopass_kernel<INV, PASS, false, false>;
  // the side of the column pass that does not meet the row pass
  if (PASS == 0 && !ntt_aligned(INV ? args.dst : args.src, INV ? args.dst_poly_stride : args.src_poly_stride,
                                args.n_polys, 2))
    kernel = ntt_twopass_kernel<INV, PASS, true, PASS == 0>;
  return launch_kernel(ctx.use_pdl, kernel, dim3(grid), dim3(kTpThreads), 0, ctx.stream, args,
                       INV ? ctx.d_row_itw : ctx.d_row_tw, job0);
}

}  // namespace

int launch_ntt_twopass(const Context &ctx, const NttArgs &args, bool inverse) {
  const int total = args.n_limbs * args.n_polys;
  for (int job0 = 0; job0 < total; job0 += kChunkJobs) {
    const int cnt = total - job0 < kChunkJobs ? total - job0 : kChunkJobs;
    if (inverse) {
      CFHE_CUDA((launch_pass<true, 1>(ctx, args, job0, cnt)));
      CFHE_CUDA((launch_pass<true, 0>(ctx, args, job0, cnt)));
    } else {
      CFHE_CUDA((launch_pass<false, 0>(ctx, args, job0, cnt)));
      CFHE_CUDA((launch_pass<false, 1>(ctx, args, job0, cnt)));
    }
  }
  CFHE_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace cfhe
