// dataterm.cuh -- host launchers of the batched data-term kernels.
#pragma once

#include "engine.cuh"

namespace gcfg {

constexpr int NBINS = 4096;                   // 16^3 colour bins per class

// Blocks of the per-image passes (histogram / sigma, extraction): each takes a
// chunk of consecutive pixels (row-major) of one image, the image's last chunk
// is shorter.  The chunk's size goes by the pixels of the whole pass: few
// pixels make few blocks, and the pass then takes as long as one block.
// Histogram / sigma pass at 1K / 2K / 4K pixels per chunk, one image (CUDA
// events, launch included): 256x256 8.6 / 11.0 / 12.7 us, 900x900 12.2 / 11.3 /
// 14.9, 1920x1080 16.4 / 14.8 / 16.8, 4096x4096 80 / 61 / 46; extraction
// 6.1 / 6.1 / 6.1, 6.1 / 6.1 / 6.1, 8.2 / 7.2 / 6.5, 25 / 18 / 14.
// 4K / 8K: 4096x4096 46 / 49, 256 uneven images of 47 million pixels 116 / 108,
// their extraction 41 / 37.
constexpr int CHUNK_PX = 8192;  // the largest chunk
inline int chunk_px_for(long long px) {
    return px <= (1 << 18) ? 1024 : px <= (1 << 22) ? 2048 : px <= (1 << 24) ? 4096 : CHUNK_PX;
}
// Chunks of any pass of at most n images and px pixels, whatever its own size
// (a pass of fewer pixels may have smaller chunks: p <= 2^24 pixels make
// p / 4096 <= p / CHUNK_PX + 2048 of them, and p <= 2^22 at most 2048).
static_assert(CHUNK_PX == 8192, "max_chunks");
inline long long max_chunks(long long n, long long px) { return px / CHUNK_PX + 2048 + n + 1; }
inline long long image_chunks(int W, int H, int chunk) { return ((long long)W * H + chunk - 1) / chunk; }

// Device buffers of the data term for a batch (per image: 2*4096 histogram
// bins, 4096 (dp, dn) entries).
struct DtArgs {
    int n_img;                // images of this pass (local index k)
    const int *ilist;         // local image k -> image (slot) index; NULL: k itself
    long long total_chunks;
    const uint8_t *rgb;       // packed row-major RGB of all images
    const uint8_t *scrib;     // packed row-major scribbles (0 none, 1 fg, 2 bg)
    const ImgDesc *img;
    ImgState *ist;
    const int2 *chunk_map;    // per chunk of the pass: (image index, chunk index within the image)
    int chunk;                // pixels per chunk
    int *hist;
    int2 *tl_lut;             // per bin the t-links (dp, dn): one 8-byte gather per pixel
    double *raw_dp, *raw_dn;  // optional (NULL): pre-rounding per-bin values
};

gcfg_status dt_tables(const DtArgs &a, cudaStream_t st);
gcfg_status dt_build(const Batch &b, const DtArgs &a, cudaStream_t st);
gcfg_status dt_apply_tlinks(const DtArgs &a, long long n, int *dp, int *dn, cudaStream_t st);
gcfg_status dt_apply_nlinks(const DtArgs &a, int W, int H, int *up, int *down, int *left, int *right,
                            cudaStream_t st);

}  // namespace gcfg
