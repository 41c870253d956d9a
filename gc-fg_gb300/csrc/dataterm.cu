// dataterm.cu -- colour-histogram t-links, contrast-sensitive n-links and
// the fused image -> tile-space residual graph build, for a whole batch.
//
// Replaces the reference's data-term module (DataTerm.cpp:52-205,
// DataTermKernels.cu:19-150), whose Gaussian KDE over a 256^3 cube is
// replaced by a 16^3 colour histogram per class:
//   p_k(bin) = (H_k[bin] + 1) / (N_k + 4096),  bin = (r>>4, g>>4, b>>4)
//   dp = round(10 * -log p_bg)   (source / foreground t-link)
//   dn = round(10 * -log p_fg)   (sink / background t-link)
// N-links: w = round(lambda * exp(-||dI||^2 / (2 sigma^2))), sigma^2 = mean
// ||dI||^2 over all horizontally and vertically adjacent pairs.  The
// reference has no n-link kernel; its callers pass per-direction arrays
// (solveMRF.cu:87-90) that InitGraphVarEdges consumes
// (GraphCutKernels.cu:165-214).
//
// Exactness: the CPU oracle evaluates these expressions in double precision.
// Here the 4096 per-bin t-links of an image go into a table, and the n-link
// of every pixel pair is evaluated directly; both use a float evaluation
// whenever it is provably far from a rounding boundary and the oracle's
// double expression otherwise, so every int32 capacity matches bit for bit.
#include <cstring>

#include "dataterm.cuh"

namespace gcfg {

__device__ __forceinline__ int color_bin3(const uint8_t *__restrict__ p) {
    return ((p[0] >> 4) << 8) | ((p[1] >> 4) << 4) | (p[2] >> 4);
}

// Colour of a pixel as one word: r | g << 8 | b << 16.
__device__ __forceinline__ uint32_t pack_rgb(const uint8_t *__restrict__ p) {
    return (uint32_t)__ldg(p) | ((uint32_t)__ldg(p + 1) << 8) | ((uint32_t)__ldg(p + 2) << 16);
}

// ||a - b||^2 of two packed colours: per-byte absolute differences, then the
// dot product of that word with itself (the top byte is 0 in both).
__device__ __forceinline__ int diff2w(uint32_t a, uint32_t b) {
    const uint32_t d = __vabsdiffu4(a, b);
    return (int)__dp4a(d, d, 0u);
}

__device__ __forceinline__ int color_binw(uint32_t c) {
    return (((c >> 4) & 0xFu) << 8) | (((c >> 12) & 0xFu) << 4) | ((c >> 20) & 0xFu);
}

// ---------------------------------------------------------------------------
// Quantised table entries.  The reference value is the double expression
// the CPU oracle evaluates; a float evaluation decides the rounding whenever
// it lies farther from a .5 boundary than its proven error, and the double
// expression is evaluated only for the near-ties that remain.
// ---------------------------------------------------------------------------

// 10 * -ln((h + 1) / N) in double (the oracle's expression).  Not inlined,
// so that the compiler cannot speculate it into the float fast path.
__device__ __noinline__ double tlink_raw(int h, long long N) {
    const double p = (double)(h + 1) / (double)N;
    return 10.0 * -log(p);
}

// round(10 * -ln((h+1)/N)).  Float error: the ratio carries <= 3 ulp
// (conversions and division, 1.8e-7 relative), which moves the log by
// <= 1.8e-7; logf adds <= 1 ulp of a result <= 22 (1.9e-6); times 10, and
// half an ulp of the product (7.6e-6): < 3e-5.  Margin used: 1e-4, as a warp
// with one entry inside it runs the double expression on a pipe of two lanes
// per SM and cycle, which bounds the tables' kernel: 256 images 36 us with
// a margin of 1e-3, 18 with 1e-4.
__device__ __forceinline__ int tlink_quant(int h, long long N) {
    const float pf = (float)(h + 1) / (float)N;
    const float v = -10.0f * logf(pf);
    const float fr = v - floorf(v);
    if (fabsf(fr - 0.5f) > 1e-4f) return (int)floorf(v + 0.5f);
    return (int)round(tlink_raw(h, N));
}

// round(lambda * exp(-d2 / (2 s2))).  The fast path evaluates
// v = lf * 2^z, z = -d2 * scale, scale = (float)(log2(e) / (2 s2)), with one
// ex2.approx.ftz.f32 (the hardware base-2 exponential; PTX documents a
// maximum relative error of about 2^-22, and gcfg_selftest_ex2 measures it
// over [-64, 0] on the device, where the tests require <= 2^-21).  Error of
// v: d2 is exact; scale and the product round once each, so z is off by
// <= 2^-23 |z|, i.e. 2^z by a relative 1.2e-7 |a| with a = z ln 2 the
// natural exponent; ex2 adds <= 2^-21 (4.8e-7); lf = (float)lambda and the
// final product <= 0.5 ulp each (1.2e-7): v is off by < v * (1.2e-7 |a| +
// 7.2e-7).  A wrong rounding needs v within that error of some k + 0.5,
// where v <= lambda and |a| = ln(lambda / (k + 0.5)) <= ln(2 lambda): the
// error is then < lambda * (1.2e-7 ln(2 lambda) + 7.2e-7).  The margin used
// is about twice that: lambda * (2.5e-7 ln(2 lambda + 1) + 1.5e-6) + 1e-6,
// set per image.  Within the margin the double expression decides.  (Large
// |a| only make v smaller: it underflows toward 0 and rounds to 0.)
//
// The fast path uses no conversion instructions (they share a slow pipe on
// this GPU): d2 < 2^23 becomes a float by writing it into the mantissa of
// 2^23, and for lambda < 2^22 the nearest integer of v comes from adding
// 1.5 * 2^23 (round to nearest even; exact ties cannot pass the margin test).
// v is at distance 0.5 - |v - rint(v)| from the nearest k + 0.5, so the
// margin test reads |v - rint(v)| < 0.5 - margin.
struct NlinkParams {
    float lf, scale;     // (float)lambda, (float)(log2(e) / (2 sigma^2))
    float margin;        // per image, from the error bound above
    float half_margin;   // 0.5 - margin
    int small;           // lambda < 2^22: the magic-number rounding applies
    int constant;        // constant image: every weight is const_w = round(lambda)
    int const_w;
    double lambda, s2;   // only read on the exact (near-tie) path
};

// round(lambda * exp(-d2 / (2 s2))) in double: the oracle's expression.  Not
// inlined, so that it cannot be speculated into the float fast path.
__device__ __noinline__ int nlink_exact(int d2, double lambda, double s2) {
    const double a = -(double)d2 / (2.0 * s2);
    return (int)round(lambda * exp(a));
}

// sigma^2 and the n-link constants of image im, from its sigma_sum.
__device__ __forceinline__ void img_params(const ImgDesc *__restrict__ img, ImgState *ist, int im) {
    const unsigned long long s = ist[im].sigma_sum;
    const long long count = (long long)(img[im].W - 1) * img[im].H + (long long)img[im].W * (img[im].H - 1);
    const double s2 = (s == 0 || count == 0) ? 0.0 : (double)s / (double)count;
    ist[im].s2 = s2;
    ist[im].ex2_scale = s2 > 0.0 ? (float)(1.4426950408889634 / (2.0 * s2)) : 0.f;  // log2(e) / (2 s2)
    ist[im].lambda_f = (float)img[im].lambda;
    ist[im].const_w = (int)round(img[im].lambda);
    const double lam = img[im].lambda;
    ist[im].nl_margin = (float)(lam * (2.5e-7 * log(2.0 * lam + 1.0) + 1.5e-6) + 1e-6);
}

// The same for every image of a pass without scribbles (k_tlut_b otherwise
// does it beside its tables: one launch and 3 us less per call).
__global__ void k_img_params(const int *__restrict__ ilist, const ImgDesc *__restrict__ img, int n_img,
                             ImgState *ist) {
    const int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li < n_img) img_params(img, ist, ilist ? ilist[li] : li);
}

__device__ __forceinline__ NlinkParams nlink_params(double lambda, const ImgState &st) {
    NlinkParams q;
    q.lambda = lambda;
    q.s2 = st.s2;
    q.lf = st.lambda_f;
    q.scale = st.ex2_scale;
    q.constant = st.ex2_scale == 0.f;
    q.const_w = st.const_w;
    q.margin = st.nl_margin;
    q.half_margin = 0.5f - q.margin;
    q.small = q.lf < 4194304.0f;
    return q;
}

// Exact float of 0 <= d2 < 2^23 (squared colour distances are <= 3 * 255^2).
__device__ __forceinline__ float small_int_to_float(int d2) {
    return __fsub_rn(__int_as_float(0x4B000000 | d2), 8388608.0f);
}

__device__ __forceinline__ float ex2_approx(float z) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(z));
    return r;
}

// The float fast path where q.small holds (see nlink_fast).
__device__ __forceinline__ bool nlink_fast_small(int d2, const NlinkParams &q, int &w) {
    const float v = q.lf * ex2_approx(-small_int_to_float(d2) * q.scale);
    const float t = __fadd_rn(v, 12582912.0f);  // 1.5 * 2^23 + rint(v)
    w = __float_as_int(t) - 0x4B400000;
    return fabsf(__fsub_rn(v, __fsub_rn(t, 12582912.0f))) < q.half_margin;
}

// The float fast path: w = the rounded weight, true when v is farther than
// the margin from a rounding boundary (else the double expression decides).
__device__ __forceinline__ bool nlink_fast(int d2, const NlinkParams &q, int &w) {
    if (q.small) return nlink_fast_small(d2, q, w);
    const float v = q.lf * ex2_approx(-small_int_to_float(d2) * q.scale);
    const float fr = v - floorf(v);
    w = (int)floorf(v + 0.5f);
    return fabsf(fr - 0.5f) > q.margin;
}

__device__ __forceinline__ int nlink_quant(int d2, const NlinkParams &q) {
    int w;
    return nlink_fast(d2, q, w) ? w : nlink_exact(d2, q.lambda, q.s2);
}

// Aligned 32-bit word at a (a % 4 == 0) of the byte range [lo, hi): one load
// when the word lies inside, else the bytes inside and zeros elsewhere.
__device__ __forceinline__ uint32_t word_in(uintptr_t a, uintptr_t lo, uintptr_t hi) {
    if (a >= lo && a + 4 <= hi) return __ldg(reinterpret_cast<const uint32_t *>(a));
    uint32_t w = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (a + k >= lo && a + k < hi) w |= (uint32_t)__ldg(reinterpret_cast<const uint8_t *>(a + k)) << (8 * k);
    return w;
}

// The same for an aligned 16-byte vector (a % 16 == 0).
__device__ __forceinline__ uint4 vec_in(uintptr_t a, uintptr_t lo, uintptr_t hi) {
    if (a >= lo && a + 16 <= hi) return __ldg(reinterpret_cast<const uint4 *>(a));
    return make_uint4(word_in(a, lo, hi), word_in(a + 4, lo, hi), word_in(a + 8, lo, hi), word_in(a + 12, lo, hi));
}

// Bytes b of a word whose offsets o + b fall in [k0, k1) (32-bit offsets).
__device__ __forceinline__ uint32_t byte_mask(int o, int k0, int k1) {
    const int f = k0 - o, l = k1 - o;  // first and one-past-last valid byte
    const uint32_t upto_l = l <= 0 ? 0u : l >= 4 ? 0xFFFFFFFFu : (1u << (8 * l)) - 1u;
    const uint32_t upto_f = f <= 0 ? 0u : f >= 4 ? 0xFFFFFFFFu : (1u << (8 * f)) - 1u;
    return upto_l & ~upto_f;
}

__device__ __forceinline__ uint32_t sq4(uint32_t a, uint32_t b) {
    const uint32_t d = __vabsdiffu4(a, b);
    return __dp4a(d, d, 0u);
}

// Sum over the byte pairs of one chunk (see k_hist_sigma_b).  The chunk's
// bytes are offsets [0, L) relative to `c0` (its first byte); a lane takes
// the aligned 16-byte vector at aw + 16 v, v = lane, lane + 32, ...: its
// right partners (bytes + 3) come from itself and the next lane's first
// word, its down partners (bytes + 3W) from the two vectors at
// + (3W rounded down to 16) shifted by (3W mod 16) bytes: WS whole words
// and BS bytes, WS fixed per instantiation.  Byte k pairs right when
// k < kh and down when k < kv (chunk-relative).
template <int WS>
__device__ __forceinline__ uint32_t sigma_chunk(uintptr_t lo, uintptr_t hi, uintptr_t c0, uintptr_t aw, int nvec,
                                                uintptr_t vstep, int bs, int kh, int kv, uint4 *keep) {
    const int lane = threadIdx.x & 31;
    uint32_t acc = 0;  // at most 7 vectors of 32 pairs of 65025 per thread
    for (int v0 = (int)threadIdx.x - lane; v0 < nvec; v0 += blockDim.x) {  // warp-uniform trip count
        const int vi = v0 + lane;
        const uintptr_t a = aw + 16 * (uintptr_t)vi;
        // every lane loads (a lane past the end supplies its neighbour's next
        // vector); bytes outside the image read as 0
        uint4 c, u, u31 = make_uint4(0, 0, 0, 0);
        uint32_t c31 = 0;
        if (a >= lo && a + vstep + 32 <= hi) {
            c = __ldg(reinterpret_cast<const uint4 *>(a));
            u = __ldg(reinterpret_cast<const uint4 *>(a + vstep));
            if (lane == 31) {
                c31 = __ldg(reinterpret_cast<const uint32_t *>(a + 16));
                u31 = __ldg(reinterpret_cast<const uint4 *>(a + vstep + 16));
            }
        } else {
            c = vec_in(a, lo, hi);
            u = vec_in(a + vstep, lo, hi);
            if (lane == 31) {
                c31 = word_in(a + 16, lo, hi);
                u31 = vec_in(a + vstep + 16, lo, hi);
            }
        }
        uint32_t n0 = __shfl_down_sync(0xffffffffu, c.x, 1);
        uint32_t un[4];
        un[0] = __shfl_down_sync(0xffffffffu, u.x, 1);
        un[1] = WS >= 1 ? __shfl_down_sync(0xffffffffu, u.y, 1) : 0u;
        un[2] = WS >= 2 ? __shfl_down_sync(0xffffffffu, u.z, 1) : 0u;
        un[3] = WS >= 3 ? __shfl_down_sync(0xffffffffu, u.w, 1) : 0u;
        if (lane == 31) {
            n0 = c31;
            un[0] = u31.x;
            un[1] = u31.y;
            un[2] = u31.z;
            un[3] = u31.w;
        }
        if (vi < nvec) {
            keep[vi] = c;  // the chunk's colours, for the histogram pass
            const uint32_t cw[4] = {c.x, c.y, c.z, c.w};
            const uint32_t hw[5] = {c.x, c.y, c.z, c.w, n0};
            const uint32_t vw[8] = {u.x, u.y, u.z, u.w, un[0], un[1], un[2], un[3]};
            const int o = (int)(a - c0);  // chunk-relative offset of the vector's byte 0
            const bool full = o >= 0 && o + 16 <= kh && o + 16 <= kv;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t dh = __vabsdiffu4(cw[j], __funnelshift_r(hw[j], hw[j + 1], 24));
                uint32_t dv = __vabsdiffu4(cw[j], __funnelshift_r(vw[j + WS], vw[j + WS + 1], bs));
                if (!full) {
                    dh &= byte_mask(o + 4 * j, 0, kh);
                    dv &= byte_mask(o + 4 * j, 0, kv);
                }
                acc = __dp4a(dv, dv, __dp4a(dh, dh, acc));
            }
        }
    }
    return acc;
}

// Shared memory of a block for its chunk: no more than it needs, as what is
// left of the SM's is the L1 cache that serves the rows below (4096x4096, chunks
// of 4096 pixels: 46 us with 12 KB per block, 48 with 24).
inline size_t hist_smem(int chunk) { return ((3 * (size_t)chunk + 15) / 16 + 1) * sizeof(uint4); }

// One pass over a chunk of an image (`chunk` consecutive pixels, row-major):
// the exact sum of ||dI||^2 over right and down neighbour pairs (for sigma^2)
// and the scribble colour histograms (privatised per block in shared memory,
// equal bins of a warp aggregated with __match_any_sync before the shared
// atomics).
//
// The sum runs on the image's byte stream B (3 bytes per pixel, row-major):
// right pairs = sum of (B[k] - B[k + 3])^2 over the chunk's bytes k with
// k + 3 inside the image, minus the pairs that straddle a row end; down pairs
// = sum of (B[k] - B[k + 3W])^2 over the chunk's bytes above the image's last
// row.  Per 4 bytes: one __vabsdiffu4 + __dp4a for each direction.
// Eight blocks per SM (32 registers, 16 bytes of spills): the pass waits on
// memory, and the fuller SM hides more of it than six blocks with 40
// registers (batch256 0.130 -> 0.112 ms).
__global__ void __launch_bounds__(256, 8) k_hist_sigma_b(const uint8_t *__restrict__ rgb,
                                                      const uint8_t *__restrict__ scrib,
                                                      const ImgDesc *__restrict__ img,
                                                      const int2 *__restrict__ chunk_map, int chunk,
                                                      int *__restrict__ hist, ImgState *ist) {
    extern __shared__ uint4 keep[];  // the chunk's bytes from its 16-aligned start (hist_smem)
    // (image, chunk within the image); no map: one image
    const int2 cm = chunk_map ? __ldg(chunk_map + blockIdx.x) : make_int2(0, (int)blockIdx.x);
    const int im = cm.x;
    const int W = img[im].W, H = img[im].H;
    const long long npx = (long long)W * H;
    const long long p0 = (long long)cm.y * chunk;
    const int n = (int)min((long long)chunk, npx - p0);  // pixels of the chunk
    const long long pix0 = img[im].pix0;
    const uint8_t *base = rgb + 3 * pix0;
    const bool do_hist = scrib != nullptr;
    const int lane = threadIdx.x & 31;
    unsigned long long acc = 0;
    {
        const long long W3 = 3LL * W, b0 = 3 * p0;
        const uintptr_t lo = (uintptr_t)base, hi = lo + (uintptr_t)(3 * npx);
        const uintptr_t c0 = lo + (uintptr_t)b0;
        const uintptr_t aw = c0 & ~(uintptr_t)15;
        const int L = 3 * n;
        const int nvec = (int)((c0 + L - aw + 15) >> 4);
        // chunk-relative limits: k + 3 inside the image; k + 3W inside the image
        const int kh = (int)min((long long)L, 3 * npx - 3 - b0);
        const int kv = (int)max(-1LL, min((long long)L, 3 * npx - W3 - b0));
        const uintptr_t vstep = (uintptr_t)(W3 & ~15LL);
        const int rem = (int)(W3 & 15);
        const int bs = (rem & 3) * 8;
        switch (rem >> 2) {
            case 0: acc = sigma_chunk<0>(lo, hi, c0, aw, nvec, vstep, bs, kh, kv, keep); break;
            case 1: acc = sigma_chunk<1>(lo, hi, c0, aw, nvec, vstep, bs, kh, kv, keep); break;
            case 2: acc = sigma_chunk<2>(lo, hi, c0, aw, nvec, vstep, bs, kh, kv, keep); break;
            default: acc = sigma_chunk<3>(lo, hi, c0, aw, nvec, vstep, bs, kh, kv, keep); break;
        }
        // right pairs that straddle a row end: rows y whose last pixel lies in
        // the chunk, below which another row follows
        const long long ya = (p0 + W) / W - 1, yb = min((p0 + n) / W - 1, (long long)H - 2);
        for (long long y = ya + threadIdx.x; y <= yb; y += blockDim.x) {
            const long long e = (y + 1) * W;  // first pixel of row y + 1
            acc -= sq4(pack_rgb(base + 3 * (e - 1)), pack_rgb(base + 3 * e));
        }
    }
    if (do_hist) {
        __syncthreads();  // the kept colours
        const uint8_t *kb = reinterpret_cast<const uint8_t *>(keep) + (int)(((uintptr_t)base + 3 * p0) & 15);
        int *dst = hist + (size_t)im * 2 * NBINS;
        // The chunk's scribble bytes, one aligned word per lane (128 pixels per
        // warp and step, so that a fully marked chunk is shared by all warps:
        // with 16 bytes per lane and the list for every step, the border strip's
        // chunks took the pass of a 256x256 image 17 us, of 1920x1080 20 us;
        // 8.6 and 14.8 this way, launch included).
        // Equal bins of a round add once, with a fire-and-forget global add.
        // Where half the step's pixels are marked (rows of a strip), round j
        // takes byte j of every lane; otherwise (ends of strips, squares) the
        // warp lists its marked bytes by a prefix sum of the lanes' counts and
        // bins them 32 per round, lane k taking item k of the list.
        const uintptr_t slo = (uintptr_t)(scrib + pix0), shi = slo + (uintptr_t)npx;
        const uintptr_t s0 = slo + (uintptr_t)p0;
        const uintptr_t saw = s0 & ~(uintptr_t)3;
        const int nsw = (int)((s0 + n - saw + 3) >> 2);
        auto bin = [&](bool on, int px, int cls) {  // pixel px of the chunk, class 1 or 2
            int key = -1;
            if (on) {
                const uint32_t col = (uint32_t)kb[3 * px] | ((uint32_t)kb[3 * px + 1] << 8) |
                                     ((uint32_t)kb[3 * px + 2] << 16);
                key = (cls - 1) * NBINS + color_binw(col);
            }
            const unsigned same = __match_any_sync(0xffffffffu, key);
            if (on && lane == __ffs(same) - 1) atomicAdd(dst + key, __popc(same));
        };
        for (int v0 = (int)threadIdx.x - lane; v0 < nsw; v0 += blockDim.x) {
            const int vi = v0 + lane;
            const uintptr_t a = saw + 4 * (uintptr_t)vi;
            uint32_t w;
            if (saw + 4 * (uintptr_t)v0 >= slo && saw + 4 * (uintptr_t)(v0 + 32) <= shi)  // warp-uniform
                w = __ldg(reinterpret_cast<const uint32_t *>(a));
            else
                w = vi < nsw ? word_in(a, slo, shi) : 0u;
            if (!__any_sync(0xffffffffu, w != 0)) continue;  // most of the image
            const int o = (int)(a - s0);  // chunk pixel of the word's byte 0
            // bit b: byte b is 1 or 2 and lies in the chunk
            unsigned todo = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const uint32_t v = (w >> (8 * b)) & 0xFFu;
                todo |= (unsigned)(v - 1u < 2u && o + b >= 0 && o + b < n) << b;
            }
            const int cnt = __popc(todo);
            if (!__any_sync(0xffffffffu, cnt != 0)) continue;
            const int total = (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
            if (total >= 64) {  // warp-uniform
#pragma unroll
                for (int b = 0; b < 4; ++b) bin((todo >> b) & 1u, o + b, (int)((w >> (8 * b)) & 0xFFu));
                continue;
            }
            int incl = cnt;  // inclusive prefix sum of the counts over the warp
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += v;
            }
            for (int r0 = 0; r0 < total; r0 += 32) {  // warp-uniform
                const int k = r0 + lane;
                // owner: the first lane whose inclusive sum exceeds k
                int own = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1) {
                    const int probe = __shfl_sync(0xffffffffu, incl, own + step - 1);
                    if (probe <= k) own += step;
                }
                unsigned om = __shfl_sync(0xffffffffu, todo, own);
                const int oincl = __shfl_sync(0xffffffffu, incl, own);
                const int oo = __shfl_sync(0xffffffffu, o, own);
                const uint32_t ow = __shfl_sync(0xffffffffu, w, own);
                // the (k - owner's exclusive sum)-th of the owner's at most four marked bytes
                const int skip = k - (oincl - __popc(om));
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (q < skip) om &= om - 1;
                const int b = __ffs(om) - 1;
                bin(k < total, oo + b, (int)((ow >> (8 * b)) & 0xFFu));
            }
        }
    }
    warp_atomic_add_u64(&ist[im].sigma_sum, acc);
}

// Per-bin t-link tables (one block per image, double precision), and the
// image's n-link constants by the block's last thread.
__global__ void __launch_bounds__(1024) k_tlut_b(const int *__restrict__ ilist, const int *hist,
                                                 const ImgDesc *__restrict__ img, ImgState *ist,
                                                 int2 *__restrict__ tl_lut,
                                                 double *raw_dp, double *raw_dn) {
    __shared__ long long part[2][32];
    cudaGridDependencySynchronize();
    const int im = ilist ? ilist[blockIdx.x] : blockIdx.x;
    if (threadIdx.x == blockDim.x - 1) img_params(img, ist, im);
    const int *hf = hist + (size_t)im * 2 * NBINS;
    const int *hb = hf + NBINS;
    long long nf = 0, nb = 0;
    for (int b = threadIdx.x; b < NBINS; b += blockDim.x) {
        nf += hf[b];
        nb += hb[b];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nf += __shfl_down_sync(0xffffffffu, nf, o);
        nb += __shfl_down_sync(0xffffffffu, nb, o);
    }
    if ((threadIdx.x & 31) == 0) {
        part[0][threadIdx.x >> 5] = nf;
        part[1][threadIdx.x >> 5] = nb;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        nf = threadIdx.x < (blockDim.x >> 5) ? part[0][threadIdx.x] : 0;
        nb = threadIdx.x < (blockDim.x >> 5) ? part[1][threadIdx.x] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            nf += __shfl_down_sync(0xffffffffu, nf, o);
            nb += __shfl_down_sync(0xffffffffu, nb, o);
        }
        if (threadIdx.x == 0) {
            part[0][0] = nf;
            part[1][0] = nb;
        }
    }
    __syncthreads();
    const long long Nf = part[0][0] + NBINS, Nb = part[1][0] + NBINS;
    for (int b = threadIdx.x; b < NBINS; b += blockDim.x) {
        int qdp, qdn;
        if (raw_dp || raw_dn) {
            const double rdp = tlink_raw(hb[b], Nb), rdn = tlink_raw(hf[b], Nf);
            qdp = (int)round(rdp);
            qdn = (int)round(rdn);
            if (raw_dp) raw_dp[(size_t)im * NBINS + b] = rdp;
            if (raw_dn) raw_dn[(size_t)im * NBINS + b] = rdn;
        } else {
            qdp = tlink_quant(hb[b], Nb);
            qdn = tlink_quant(hf[b], Nf);
        }
        tl_lut[(size_t)im * NBINS + b] = make_int2(qdp, qdn);
    }
}

// N-link weight of a pair at squared colour distance d2 (s2 = sigma^2,
// 0 for a constant image, whose weights are all lambda).
__device__ __forceinline__ int nlink_w(int d2, const NlinkParams &q) {
    return q.constant ? q.const_w : nlink_quant(d2, q);
}

// Fused image -> residual graph of one tile: t-link gather, n-links, the
// reference's interior/border conventions, tile-major output.
//
// A warp walks down a strip of rows, lane = column, and needs no other warp's
// results: each lane reads its pixel and the one to the right as aligned words
// (every line of the image's rows comes from L1 after the first of them), keeps
// the row below's colour for the next row, and weighs the edges to the right
// and down; the weight from the left comes from the next lane, that from above
// from the row before.  A strip reads one row above and one below it again and
// weighs the edges over its upper border a second time (the weight is symmetric
// in its two pixels).  An edge that touches the 1-pixel image border has
// capacity 0, as in the reference's graph (GraphCutKernels.cu:112-214).
//
// What bounds it: the instructions issued and, beside them, the shared-memory
// and L1 pipe (a gather of random bins is up to 32 lines).  Staging the tile's
// colours, then weighing all edges, then joining them, with a barrier between,
// took 8300 warp instructions per tile; inside the image a strip needs none of
// the border's checks and, with one 8-byte gather for both t-links, about
// 4000.  256 uneven images (54,000 tiles) 420 -> 330 us, 4096x4096 135 -> 96
// (400 MB at 4.2 TB/s), 1920x1080 23.6 -> 19.1.
struct BuildTile {
    int W, H, x, ys;        // image size, the lane's column, the strip's first row
    const uint8_t *base;    // the image's first byte
    const int2 *lut;
    int4 *cap;              // the strip's first row in the arena, this lane's column
    int *exc;
    uint32_t (*msk)[TILE_H];
    int r0;                 // the strip's first row within the tile
};

// What a tile needs.  INNER: the tile and the pixels around it lie inside the
// 1-pixel border, so that no pixel, byte or edge needs a check (nine tenths of
// the tiles of 1920x1080, half of those of 256x256).  EDGE: they do not.  Both:
// the image's byte offsets fit 32 bits, lambda < 2^22 (q.small) and the image
// is not constant.  ANY: everything else.
enum { BUILD_INNER, BUILD_EDGE, BUILD_ANY };
template <int KIND, int STRIP>
__device__ __forceinline__ void build_strip(const BuildTile &g, const NlinkParams &q, uint32_t &idp, uint32_t &rinit,
                                            uint32_t &pos) {
    constexpr bool INNER = KIND == BUILD_INNER;
    const int lane = threadIdx.x & 31;
    const int W = g.W, H = g.H, x = g.x;
    const uintptr_t lo = (uintptr_t)g.base, hi = lo + 3 * (uintptr_t)W * (uintptr_t)H;
    const int mis = (int)(lo & 3);
    const uint8_t *abase = g.base - mis;  // 4-byte aligned
    // The three aligned words that hold pixel (px, y) and its right neighbour,
    // and the place of its first byte in them (mod 4).  Where they reach past
    // the pair they stay inside the image for an inner tile; elsewhere bytes
    // outside the image, and pixels outside it, read as 0.
    struct Words {
        uint32_t w[3];
        unsigned o;
    };
    auto fetch = [&](int px, int y) {
        Words f;
        const bool in = INNER || (px >= 0 && px < W && y >= 0 && y < H);
        if (KIND != BUILD_ANY) {
            const int o = mis + 3 * (y * W + px), a = o & ~3;
            const uint8_t *p = abase + a;
            if (INNER || (in && a >= mis && a + 12 <= mis + 3 * W * H)) {
#pragma unroll
                for (int i = 0; i < 3; ++i) f.w[i] = __ldg(reinterpret_cast<const uint32_t *>(p) + i);
            } else {
#pragma unroll
                for (int i = 0; i < 3; ++i) f.w[i] = in ? word_in((uintptr_t)p + 4 * i, lo, hi) : 0u;
            }
            f.o = (unsigned)o;
        } else {
            const uintptr_t a = in ? lo + 3 * ((uintptr_t)y * W + px) : hi + 4;
#pragma unroll
            for (int i = 0; i < 3; ++i) f.w[i] = word_in((a & ~(uintptr_t)3) + 4 * i, lo, hi);
            f.o = (unsigned)a;
        }
        return f;
    };
    auto cut = [](const Words &f, uint32_t &c, uint32_t &n) {  // the pair's colours
        const uint32_t a = __funnelshift_r(f.w[0], f.w[1], f.o * 8), b = __funnelshift_r(f.w[1], f.w[2], f.o * 8);
        c = a & 0xFFFFFFu;
        n = __funnelshift_r(a, b, 24) & 0xFFFFFFu;
    };
    // Weight of an edge between colours a and b (use: both ends are interior);
    // bad: the float path leaves it to the double expression.
    auto weigh = [&](uint32_t a, uint32_t b, bool use, bool &bad) {
        int w;
        if (KIND != BUILD_ANY) {
            bad = !nlink_fast_small(diff2w(a, b), q, w) && (INNER || use);
            return INNER || use ? w : 0;
        }
        bad = false;
        w = q.const_w;
        if (!q.constant) bad = use && !nlink_fast(diff2w(a, b), q, w);
        return use ? w : 0;
    };
    auto inside = [&](int px, int y) { return px >= 1 && px <= W - 2 && y >= 1 && y <= H - 2; };
    // the arena is no table: the next rows' gathers may go ahead of its stores
    int4 *__restrict__ cap = g.cap;
    int *__restrict__ exc = g.exc;
    const bool col_in = x >= 1 && x <= W - 2, cols_in = x >= 1 && x <= W - 3;  // the lane's and the next column

    constexpr int AHEAD = 3;  // rows of words in flight
    Words ring[AHEAD + 1];
    const Words fa = fetch(x, g.ys - 1);
    const int xl = x - lane - 1;  // the column left of the tile: lane r of 0..7 for row r
    const Words fl = fetch(xl, g.ys + (lane & (STRIP - 1)));
#pragma unroll
    for (int r = 0; r < AHEAD; ++r) ring[r] = fetch(x, g.ys + r);
    uint32_t c, n;  // this pixel and its right neighbour
    cut(ring[0], c, n);
    int wu, wl;  // the edge from above (this row's), from the left (lane r: row r's)
    {
        uint32_t a, b;
        bool bad;
        cut(fa, a, b);
        wu = weigh(a, c, inside(x, g.ys - 1) && inside(x, g.ys), bad);
        if (bad) wu = nlink_exact(diff2w(a, c), q.lambda, q.s2);
        cut(fl, a, b);
        const int y = g.ys + (lane & (STRIP - 1));
        wl = weigh(a, b, inside(xl, y) && inside(xl + 1, y), bad);
        if (bad) wl = nlink_exact(diff2w(a, b), q.lambda, q.s2);
    }
    // the reference sums max(dp, 0) over padded positions x + y * W32 < W * H
    // (GraphCut.cu:359-376, GraphCutKernels.cu:883-898); 32-bit for an inner tile (W32 < 2 W)
    const int w32 = (W + 31) & ~31;
    const int left = INNER ? W * H - x - g.ys * w32 : 0;
    unsigned mu = __ballot_sync(0xffffffffu, wu > 0);
#pragma unroll
    for (int r = 0; r < STRIP; ++r) {
        const int y = g.ys + r;
        if (r + AHEAD <= STRIP) ring[(r + AHEAD) % (AHEAD + 1)] = fetch(x, y + AHEAD);
        uint32_t cd, nd;  // the row below
        cut(ring[(r + 1) % (AHEAD + 1)], cd, nd);
        bool bad_r, bad_d;
        int wr = weigh(c, n, cols_in && y >= 1 && y <= H - 2, bad_r);
        int wd = weigh(c, cd, col_in && y >= 1 && y <= H - 3, bad_d);
        if (__any_sync(0xffffffffu, bad_r || bad_d)) {  // rare
            if (bad_r) wr = nlink_exact(diff2w(c, n), q.lambda, q.s2);
            if (bad_d) wd = nlink_exact(diff2w(c, cd), q.lambda, q.s2);
        }
        const int wl_r = __shfl_sync(0xffffffffu, wl, r);
        int4 k;
        k.x = __shfl_up_sync(0xffffffffu, wr, 1);
        if (lane == 0) k.x = wl_r;
        k.y = wr;
        k.z = wu;
        k.w = wd;
        int e = 0;
        if (INNER || (x < W && y < H)) {
            const int2 v = g.lut[color_binw(c)];
            const bool counted = INNER ? r * w32 < left : (long long)x + (long long)y * w32 < (long long)W * H;
            if (counted) rinit += (unsigned)max(v.x, 0);
            if (INNER || inside(x, y)) {
                e = v.x - v.y;
                idp += (unsigned)v.x;
            }
        }
        cap[r * 32] = k;
        exc[r * 32] = e;
        pos += (unsigned)max(e, 0);
        // of the six mask planes, the left one is the right one moved by a
        // column, the upper one the lower one of the row before
        const unsigned mr = __ballot_sync(0xffffffffu, wr > 0), md = __ballot_sync(0xffffffffu, wd > 0);
        const unsigned mn = __ballot_sync(0xffffffffu, e < 0), mp = __ballot_sync(0xffffffffu, e > 0);
        if (lane == 0) {
            g.msk[0][g.r0 + r] = mr << 1 | (k.x > 0 ? 1u : 0u);
            g.msk[1][g.r0 + r] = mr;
            g.msk[2][g.r0 + r] = mu;
            g.msk[3][g.r0 + r] = md;
            g.msk[4][g.r0 + r] = mn;
            g.msk[5][g.r0 + r] = mp;
        }
        mu = md;
        wu = wd;
        c = cd;
        n = nd;
    }
}

// Strips of 8 rows (4 warps per tile) do the least work per tile; up to
// BUILD_SMALL_TILES tiles, which are all resident at once, the time is that of
// one strip, and strips of 4 rows are shorter: 8 against 4 warps 9.7 / 11.9 us
// for 256x256 (64 tiles), 10.1 / 13.9 for 512x512, 12.2 / 12.5 for 900x900 (841
// tiles), 20.1 / 19.5 for 1920x1080 (2040), 121 / 96 for 4096x4096.  (2 rows: 8.7
// for 256x256, 14.3 for 900x900; 16 rows: 100 for 4096x4096, 396 for the batch.)
constexpr int BUILD_SMALL_TILES = 1024;
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 32 / WARPS) k_build_img_b(Batch b, const uint8_t *__restrict__ rgb,
                                                                   const int2 *tl_lut) {
    constexpr int STRIP = TILE_H / WARPS;
    __shared__ uint32_t msk[6][TILE_H];  // mask planes of the tile, stored coalesced below
    __shared__ unsigned long long wsum[3][WARPS];
    cudaGridDependencySynchronize();
    const int t = batch_tile(b, blockIdx.x);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int im = __ldg(b.tile_img + t);
    const ImgDesc &d = b.img[im];
    const int W = d.W, H = d.H, tiles_x = d.tiles_x, tiles_y = d.tiles_y;
    const int lt = t - d.tile0;
    const int ty = lt / tiles_x, tx = lt - ty * tiles_x;
    if (threadIdx.x == 0)  // the tile's neighbours, for the solver
        b.tile_nb[t] = make_int4(tx > 0 ? t - 1 : -1, tx < tiles_x - 1 ? t + 1 : -1, ty > 0 ? t - tiles_x : -1,
                                 ty < tiles_y - 1 ? t + tiles_x : -1);
    const int x0 = tx * TILE_W, y0 = ty * TILE_H;
    const NlinkParams q = nlink_params(d.lambda, b.ist[im]);
    BuildTile g;
    g.W = W;
    g.H = H;
    g.x = x0 + lane;
    g.r0 = STRIP * warp;
    g.ys = y0 + g.r0;
    g.base = rgb + 3 * d.pix0;
    g.lut = tl_lut + (size_t)im * NBINS;
    g.cap = b.cap + (size_t)t * TPX + g.r0 * 32 + lane;
    g.exc = b.exc + (size_t)t * TPX + g.r0 * 32 + lane;
    g.msk = msk;
    uint32_t idp = 0, rinit = 0, pos = 0;
    if (3LL * W * H >= (1LL << 30) || !q.small || q.constant)
        build_strip<BUILD_ANY, STRIP>(g, q, idp, rinit, pos);
    else if (tx > 0 && ty > 0 && x0 + TILE_W + 1 < W && y0 + TILE_H + 1 < H)
        build_strip<BUILD_INNER, STRIP>(g, q, idp, rinit, pos);
    else
        build_strip<BUILD_EDGE, STRIP>(g, q, idp, rinit, pos);
    // Per-thread sums stay below 2^31 (8 pixels of at most GCFG_MAX_CAP), so
    // they are 32-bit and each warp adds them exactly with two 32-bit
    // reductions of their 16-bit halves.
    {
        const uint32_t v[3] = {idp, rinit, pos};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const unsigned long long l = __reduce_add_sync(0xffffffffu, v[k] & 0xFFFFu);
            const unsigned long long h = __reduce_add_sync(0xffffffffu, v[k] >> 16);
            if (lane == 0) wsum[k][warp] = (h << 16) + l;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 6 * TILE_H; i += WARPS * 32)
        b.tmask[(size_t)t * 6 * 32 + i] = msk[i >> 5][i & 31];
    if (warp == 0) {
        // lanes 0..2: the tile's three sums
        unsigned long long tot = 0;
        if (lane < 3)
            for (int w = 0; w < WARPS; ++w) tot += wsum[lane][w];
        if (lane == 0 && tot) atomicAdd(&b.ist[im].interior_dp, tot);
        if (lane == 1 && tot) atomicAdd(&b.ist[im].ref_init, tot);
        if (lane == 2) b.tile_pos[t] = tot;
    }
}

// Row-major t-link / n-link arrays of image 0 (the stand-alone data-term API).
__global__ void k_tlinks_apply(const uint8_t *__restrict__ rgb, long long n,
                               const int2 *__restrict__ tl_lut, int *__restrict__ dp, int *__restrict__ dn) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int bin = color_bin3(rgb + 3 * i);
    const int2 v = __ldg(tl_lut + bin);
    dp[i] = v.x;
    dn[i] = v.y;
}

// One block per 32 x 32 pixels, thread (x, y) four rows of column x.  Each
// edge is weighed once, by its left or upper pixel, which writes it to both
// pixels' arrays; colours are read once per row, the right neighbour's and the
// row below's come from the next lane and the next row.  (One thread per pixel
// that weighed its four edges itself, and so each edge twice, from byte loads:
// 17.3 us for 1279x853, 10.8 this way.)
__global__ void __launch_bounds__(256) k_nlinks_apply(const uint8_t *__restrict__ rgb,
                                                      const ImgDesc *__restrict__ img, const ImgState *ist,
                                                      int *__restrict__ up, int *__restrict__ down,
                                                      int *__restrict__ left, int *__restrict__ right) {
    constexpr int ROWS = 4;
    const ImgDesc d = img[0];
    const int W = d.W, H = d.H;
    const int lane = threadIdx.x;
    const int x = blockIdx.x * 32 + lane, y0 = (blockIdx.y * 8 + threadIdx.y) * ROWS;
    const NlinkParams q = nlink_params(d.lambda, ist[0]);
    // colours of rows y0 .. y0 + ROWS, and of the pixel right of the last lane's
    uint32_t c[ROWS + 1], cr[ROWS];
#pragma unroll
    for (int k = 0; k <= ROWS; ++k) {
        const int y = y0 + k;
        const uint8_t *p = rgb + 3 * ((long long)y * W + x);
        c[k] = x < W && y < H ? pack_rgb(p) : 0u;
        if (k < ROWS) cr[k] = lane == 31 && x + 1 < W && y < H ? pack_rgb(p + 3) : 0u;
    }
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        const int y = y0 + k;
        uint32_t r = __shfl_down_sync(0xffffffffu, c[k], 1);
        if (lane == 31) r = cr[k];
        if (x >= W || y >= H) continue;
        const long long i = (long long)y * W + x;
        const int wr = x + 1 < W ? nlink_w(diff2w(c[k], r), q) : 0;
        const int wd = y + 1 < H ? nlink_w(diff2w(c[k], c[k + 1]), q) : 0;
        right[i] = wr;
        if (x + 1 < W) left[i + 1] = wr;
        if (x == 0) left[i] = 0;
        down[i] = wd;
        if (y + 1 < H) up[i + W] = wd;
        if (y == 0) up[i] = 0;
    }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------

gcfg_status dt_tables(const DtArgs &a, cudaStream_t st) {
    // a.scrib == NULL: n-link constants only (the colour histograms need
    // scribbles); the caller has cleared the histograms
    GCFG_LAUNCH(GCFG_PK_HIST, st,
                k_hist_sigma_b<<<a.total_chunks, 256, hist_smem(a.chunk), st>>>(a.rgb, a.scrib, a.img, a.chunk_map,
                                                                                a.chunk, a.hist, a.ist));
    if (a.scrib)
        GCFG_LAUNCH(GCFG_PK_TLUT, st,
                    launch_behind(k_tlut_b, a.n_img, 1024, st, a.ilist, a.hist, a.img, a.ist, a.tl_lut, a.raw_dp,
                                  a.raw_dn));
    else
        GCFG_LAUNCH(GCFG_PK_TLUT, st,
                    k_img_params<<<div_up(a.n_img, 128), 128, 0, st>>>(a.ilist, a.img, a.n_img, a.ist));
    GCFG_CK(cudaGetLastError());
    return GCFG_OK;
}

gcfg_status dt_build(const Batch &b, const DtArgs &a, cudaStream_t st) {
    const int tiles = batch_ntiles(b);
    if (tiles <= BUILD_SMALL_TILES)
        GCFG_LAUNCH(GCFG_PK_BUILD, st, launch_behind(k_build_img_b<8>, tiles, 256, st, b, a.rgb, a.tl_lut));
    else
        GCFG_LAUNCH(GCFG_PK_BUILD, st, launch_behind(k_build_img_b<4>, tiles, 128, st, b, a.rgb, a.tl_lut));
    GCFG_CK(cudaGetLastError());
    return GCFG_OK;
}

gcfg_status dt_apply_tlinks(const DtArgs &a, long long n, int *dp, int *dn, cudaStream_t st) {
    GCFG_LAUNCH(GCFG_PK_OTHER, st,
                k_tlinks_apply<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a.rgb, n, a.tl_lut, dp, dn));
    GCFG_CK(cudaGetLastError());
    return GCFG_OK;
}

gcfg_status dt_apply_nlinks(const DtArgs &a, int W, int H, int *up, int *down, int *left, int *right,
                            cudaStream_t st) {
    dim3 blk(32, 8), grd(div_up(W, 32), div_up(H, 32));
    GCFG_LAUNCH(GCFG_PK_OTHER, st,
                k_nlinks_apply<<<grd, blk, 0, st>>>(a.rgb, a.img, a.ist, up, down, left, right));
    GCFG_CK(cudaGetLastError());
    return GCFG_OK;
}

// Largest relative error of ex2_approx against the double 2^z over n
// evenly spaced z in [-64, 0] (the n-link fast path's error bound assumes
// <= 2^-21).  Relative errors are non-negative floats, so their bit
// patterns order like the values and an integer atomicMax finds the largest.
__global__ void k_selftest_ex2(long long n, int *max_bits) {
    float worst = 0.f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float z = -64.0f * (float)((double)i / (double)n);
        const double ref = exp2((double)z);
        const double rel = fabs((double)ex2_approx(z) - ref) / ref;
        worst = fmaxf(worst, (float)rel);
    }
    atomicMax(max_bits, __float_as_int(worst));
}

}  // namespace gcfg

extern "C" gcfg_status gcfg_selftest_ex2(int64_t samples, float *max_rel_err) {
    using namespace gcfg;
    if (samples < 1 || !max_rel_err) return GCFG_ERR_INVALID;
    int *d = nullptr;
    if (cudaMalloc(&d, sizeof(int)) != cudaSuccess) return GCFG_ERR_OOM;
    int bits = 0;
    cudaError_t e = cudaMemset(d, 0, sizeof(int));
    if (e == cudaSuccess) {
        k_selftest_ex2<<<1024, 256>>>((long long)samples, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&bits, d, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return GCFG_ERR_CUDA;
    memcpy(max_rel_err, &bits, sizeof(float));
    return GCFG_OK;
}
