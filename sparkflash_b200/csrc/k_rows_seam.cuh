// What the seam kernels of the layered decoders share (k_rows.cu, many rows k_rows_seam_many.cu: one residual; k_rows_streams.cu: several streams of it).
#pragma once
#include "k_rows.cuh"

namespace sfb {
namespace rows {

// one residual (k_rows.cu, k_rows_seam_many.cu)
struct SeamArgs {
  float* x;                 // [rows, d] residual, 32-bit
  const void* y;            // [rows, d] sublayer output (T) or null: no residual update
  const void* y2;           // second branch (T) or null
  const float *mw, *mw2;    // RMS weights of the two branches
  const float* parts_w;     // [rows, parts]: y is [rows, parts, d] and the output their weighted sum; or null
  const float *pw, *pb;     // post-norm (pb null: no bias), or the scale
  const void* embed;        // [vocab, d] (T)
  const int* tokens;        // [rows]
  const float* step_vec;    // [d] or null: added after the update
  float* tap;               // [rows, d] or null: the residual right after the update
  const float *nw, *nb;     // next norm, or null: h is the residual itself
  void* h;                  // [rows, d] (T) its output, or null
  const int* row_map;       // null: row = block; otherwise the residual row of output row `block`
  const float* cw;          // [taps, d] input convolution, or null
  void* hist;               // [slots, taps - 1, d] (T)
  const int *src, *dst;     // [rows] state versions of single-row segments
  int from_embed, add_embed, taps, d, vocab;
  int parts, post, rms;     // post: POST_*; rms: the next norm is an RMS norm
  float eps, embed_scale;
  Status* status;
};

constexpr int POST_LAYER = 0, POST_RMS = 1, POST_SCALE = 2;

// From two rows per SM on, of 2,048 elements (from 2,048 rows on 1,024) and more, the seam is the persistent kernel of k_rows_seam_many.cu.  0 or an error; -1: it
// does not take these.
constexpr int SEAM_MANY_ROWS = 297;
int seam_many(const SeamArgs& a, int n, cudaStream_t stream);

// several streams of the residual (k_rows_streams.cu, k_rows_seam_many.cu)
struct StreamArgs {
  float* x;                 // [rows, S, d] streams
  const void* y;            // [rows, d] sublayer output (T) or null: no update
  const float* parts_w;     // [rows, parts]: y is [rows, parts, d] and the output their weighted sum; or null
  const float *mix, *out;   // [S, S] from, to; [S]
  const void* embed;        // [vocab, d] (T): the row begins with it (y null)
  const int* tokens;        // [rows]
  float* tap;               // [rows, d] or null: the sum of the new streams
  const float* in;          // [S] or null: ones
  const float* nw;          // [d]
  void* h;                  // [rows, d] (T)
  const int* row_map;       // null: row = block; otherwise the residual row of output row `block`
  const float* cw;          // [taps, d] input convolution, or null
  void* hist;               // [slots, taps - 1, d] (T)
  const int *src, *dst;     // [rows] state versions of single-row segments
  int S, d, parts, taps, vocab, keep;    // keep: the streams are stored
  float eps, embed_scale;
  Status* status;
};
// two to four streams of 1,024 and more elements, as seam_many
int streams_many(const StreamArgs& a, int n, cudaStream_t stream);



// Input convolution of a step of single-row segments: o (channels c .. of a norm's output) becomes o + conv(o) over the carried inputs hs
// (null: zeros), whose next version is hd.  `ahead`: weights and carried inputs are held in registers (rw, rg: [taps][i][V]).
template <typename T, int V, int TW, int NV>
__device__ __forceinline__ void step_conv(float (&o)[V], int i, int c, int d, int W, const float* w, const T* hs, T* hd, bool ahead,
                                          const float (&rw)[TW][NV][V], const float (&rg)[TW][NV][V]) {
  // the convolution sees the norm's output at activation precision, as the many-row kernel does
  float acc[V], t[V];
#pragma unroll
  for (int k = 0; k < V; ++k) o[k] = to_f<T>(from_f<T>(o[k]));
  if (ahead) {
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = 0.f;
#pragma unroll
    for (int j = 0; j < TW; ++j) {
      if (j < W) {
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] += rw[j][i][k] * rg[j][i][k];
        if (j > 0) store_v<T, V>(hd + (size_t)(j - 1) * d + c, rg[j][i]);
      } else if (j == W) {
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] += rw[j][i][k] * o[k];
      }
    }
  } else {
    load_v<float, V>(w + (size_t)W * d + c, t);
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = t[k] * o[k];
#pragma unroll 4
    for (int j = 0; j < W; ++j) {
      float g[V];
      if (hs) load_v<T, V>(hs + (size_t)j * d + c, g);
      else {
#pragma unroll
        for (int k = 0; k < V; ++k) g[k] = 0.f;
      }
      load_v<float, V>(w + (size_t)j * d + c, t);
#pragma unroll
      for (int k = 0; k < V; ++k) acc[k] += t[k] * g[k];
      if (j > 0) store_v<T, V>(hd + (size_t)(j - 1) * d + c, g);
    }
  }
  if (W > 0) store_v<T, V>(hd + (size_t)(W - 1) * d + c, o);
#pragma unroll
  for (int k = 0; k < V; ++k) o[k] += acc[k];
}

}  // namespace rows
}  // namespace sfb
