// Host-buffer front end (opencnn_host_plan_*): device buffers for one problem size, copies and launches.  Host code only, so that it can be
// compiled and tested without a GPU.  Included by abi.cu, which declares what it uses: check_shape, shape_rule, TileRows, kMaxDevices,
//     cudaError_t forward(input, filter, output, workspace, N, C, H, W, K, precision, stream, rule)             the whole operator
//     cudaError_t transform_filter(filter, workspace, C, K, precision, stream)
//     cudaError_t convolve_rows(input, workspace, output, N, C, H, W, K, precision, stream, rows)               some rows of tiles
#pragma once
#include <cuda_runtime.h>
#include <functional>
#include <mutex>
#include <new>

#include "../../include/opencnn_b200.h"

namespace {

// The two streams on which a run copies in bands, one per direction: a pair per device, made when a plan first needs it and kept until the
// process exits.  A run has it to itself from its first copy until it has been waited for, so it waits for nothing that another plan
// enqueued.  A run that finds it taken, or that it can't be made, is in one piece: the other run and its own copies in one stream keep both
// directions busy already.  Runs of 32x64x64x56x56 and 32x128x128x28x28 in two threads take 940 us a pair so, 1090 with a pair of streams for
// each and 1160 with both in one queue (in one piece, both: 1165); with a third thread (64x128x128x14x14) 1180, 1300, 1365 (1195).
struct LinkStreams {
  std::mutex mutex;
  bool taken = false;
  cudaStream_t up = nullptr, down = nullptr;
};
LinkStreams g_link[kMaxDevices];

// With the device current.
bool take_link(LinkStreams &link) {
  std::lock_guard<std::mutex> lock(link.mutex);
  if (link.taken) return false;
  for (cudaStream_t *s : {&link.up, &link.down})
    if (!*s && cudaStreamCreateWithFlags(s, cudaStreamNonBlocking) != cudaSuccess) {
      cudaGetLastError();
      *s = nullptr;
      return false;
    }
  return link.taken = true;
}

void give_link(LinkStreams &link) {
  std::lock_guard<std::mutex> lock(link.mutex);
  link.taken = false;
}

// Host-buffer front end.  A run that is waited for does the upload of the input, the kernel and the download of the output in `bands` bands of
// tile rows, so that both directions of the host link are busy at once: the kernel of a band follows the rows that it reads (two
// more than its own), its output leaves while the next band's input arrives.  Runs that are only enqueued overlap with those of other
// plans and do better in one piece: four layers in rotation copy 88 GB/s so, 81 in bands.
struct HostPlan {
  int N, C, H, W, K, precision, bands;
  float *d_in = nullptr, *d_filt = nullptr, *d_out = nullptr, *d_ws = nullptr;
  cudaStream_t stream = nullptr;
  int device = 0;
  LinkStreams *link = nullptr;                                      // this and the events only with more than one band
  cudaEvent_t landed = nullptr, computed = nullptr, left = nullptr;
};

// What bands can hide is the shorter of the two copies, so a band is at least kBandBytes of twice that one, and its rows of one plane at
// least kBandRowBytes in a row (a strided copy is made of such pieces).  One call, us, by the number of bands (1: as one upload,
// kernel, download):
//     fp32 32x64x64x56x56     1: 1028  2: 827   4: 787   6: 787   7: 814   8: 820   12: 780 to 842
//     fp32 8x32x64x112x56     1: 401   2: 355   4: 335   6: 333   7: 335   8: 334   12: 334
//     fp32 32x256x256x14x14   1: 384   2: 303   4: 290   6: 340 (pieces of 4.2 KB)
//     fp32 32x128x128x28x28   1: 590   4: 469   6: 440   7: 399   8: 420   10: 433
//     tf32 64x64x64x56x56     1: 1918  2: 1525  4: 1390  6: 1370  7: 1386  8: 1413  12: 1500
//     bf16 16x64x64x60x90     1: 860   4: 664   6: 681   7: 685   8: 706   12: 749
//     fp32 64x100x64x33x37                      6: 782   7: 843   8: 859   12: 811
//     bf16 128x128x128x28x14                    6: 800   7: 813   8: 804   12: 776
//     bf16 40x7x192x38x38     1: 877  12: 932 (1.6 MB in, 44 MB out: nothing to hide)
// No number is the best for all; with six, ten of thirteen sizes were the same or up to 9 % faster than with twelve, and none more than 3 %
// slower.
constexpr size_t kBandBytes = 2400000, kBandRowBytes = 6u << 10;
constexpr int kMaxBands = 6;
int band_count(int N, int C, int H, int W, int K) {
  const size_t row = (size_t)W * N * 4, bytes = 2 * row * H * (C < K ? C : K);
  const int tile_rows = (H + 1) / 2;
  long long bands = (long long)(bytes / kBandBytes);
  if (bands > (long long)(row * H / kBandRowBytes)) bands = (long long)(row * H / kBandRowBytes);
  if (bands > tile_rows) bands = tile_rows;
  if (bands > kMaxBands) bands = kMaxBands;
  if (row * H > 0x7fffffffu) bands = 1;            // pitch of a strided copy
  return bands < 1 ? 1 : (int)bands;
}

// Asynchronous copies need page-locked memory at both ends.
bool page_locked(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

// Rows [r0, r1) of every plane of a CHWN / KHWN tensor.
cudaError_t copy_rows(float *dst, const float *src, int planes, int r0, int r1, const HostPlan *hp, cudaMemcpyKind kind, cudaStream_t stream) {
  const size_t row = (size_t)hp->W * hp->N, pitch = row * hp->H * 4;
  if (r1 <= r0) return cudaSuccess;
  return cudaMemcpy2DAsync(dst + r0 * row, pitch, src + r0 * row, pitch, (r1 - r0) * row * 4, planes, kind, stream);
}

// Whether a band's output may be written before the next band's input is read: the arrays have nothing in common, or start at the same place,
// where an output row lies over the same row of the input, which no later band reads from there.
bool bands_apart(const float *in, size_t in_n, const float *out, size_t out_n) {
  return in == out || std::less_equal<>()(in + in_n, out) || std::less_equal<>()(out + out_n, in);
}

cudaError_t run_bands(HostPlan *hp, const float *input_host, const float *filter_host, float *output_host) {
  const LinkStreams &link = *hp->link;
  const size_t f_b = (size_t)hp->C * 9 * hp->K * 4;
  const int tile_rows = (hp->H + 1) / 2;
  // what was enqueued on the plan before must be through with the device buffers
  cudaError_t e = cudaEventRecord(hp->landed, hp->stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(link.up, hp->landed, 0);
  if (e == cudaSuccess) e = cudaMemcpyAsync(hp->d_filt, filter_host, f_b, cudaMemcpyHostToDevice, link.up);
  if (e == cudaSuccess) e = cudaEventRecord(hp->landed, link.up);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(hp->stream, hp->landed, 0);
  if (e == cudaSuccess) e = transform_filter(hp->d_filt, hp->d_ws, hp->C, hp->K, hp->precision, hp->stream);
  for (int b = 0, up_to = 0; b < hp->bands && e == cudaSuccess; ++b) {
    const int t0 = (int)((long long)tile_rows * b / hp->bands), t1 = (int)((long long)tile_rows * (b + 1) / hp->bands);
    const int need = 2 * t1 + 1 < hp->H ? 2 * t1 + 1 : hp->H, end = 2 * t1 < hp->H ? 2 * t1 : hp->H;
    e = copy_rows(hp->d_in, input_host, hp->C, up_to, need, hp, cudaMemcpyHostToDevice, link.up);
    up_to = need;
    if (e == cudaSuccess) e = cudaEventRecord(hp->landed, link.up);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(hp->stream, hp->landed, 0);
    if (e == cudaSuccess) e = convolve_rows(hp->d_in, hp->d_ws, hp->d_out, hp->N, hp->C, hp->H, hp->W, hp->K, hp->precision, hp->stream, {t0, t1 - t0});
    if (e == cudaSuccess) e = cudaEventRecord(hp->computed, hp->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(link.down, hp->computed, 0);
    if (e == cudaSuccess) e = copy_rows(output_host, hp->d_out, hp->K, 2 * t0, end, hp, cudaMemcpyDeviceToHost, link.down);
  }
  // `stream` ends where everything has: it is what is waited for, here and by the next run.  After an error, too.
  cudaError_t j = cudaEventRecord(hp->landed, link.up);
  if (j == cudaSuccess) j = cudaStreamWaitEvent(hp->stream, hp->landed, 0);
  if (j == cudaSuccess) j = cudaEventRecord(hp->left, link.down);
  if (j == cudaSuccess) j = cudaStreamWaitEvent(hp->stream, hp->left, 0);
  return e != cudaSuccess ? e : j;
}

}  // namespace

extern "C" {

int opencnn_host_plan_create(void **plan, int in_n, int in_c, int in_h, int in_w, int filt_k, int precision) {
  if (!plan) return (int)cudaErrorInvalidValue;
  *plan = nullptr;
  if (precision != OPENCNN_FP32 && precision != OPENCNN_TF32 && precision != OPENCNN_BF16) return (int)cudaErrorInvalidValue;
  cudaError_t e = check_shape(in_n, in_c, in_h, in_w, filt_k, shape_rule(precision));
  if (e != cudaSuccess) return (int)e;
  HostPlan *hp = new (std::nothrow) HostPlan;
  if (!hp) return (int)cudaErrorMemoryAllocation;
  hp->N = in_n; hp->C = in_c; hp->H = in_h; hp->W = in_w; hp->K = filt_k; hp->precision = precision;
  hp->bands = band_count(in_n, in_c, in_h, in_w, filt_k);
  const size_t in_b = (size_t)in_n * in_c * in_h * in_w * 4, f_b = (size_t)in_c * 9 * filt_k * 4;
  const size_t out_b = (size_t)in_n * filt_k * in_h * in_w * 4;
  e = cudaMalloc(&hp->d_in, in_b);
  if (e == cudaSuccess) e = cudaMalloc(&hp->d_filt, f_b);
  if (e == cudaSuccess) e = cudaMalloc(&hp->d_out, out_b);
  if (e == cudaSuccess) e = cudaMalloc(&hp->d_ws, opencnn_workspace_bytes(in_c, filt_k));
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&hp->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaGetDevice(&hp->device);
  if (hp->device < 0 || hp->device >= kMaxDevices) hp->bands = 1;
  if (hp->bands > 1) {
    for (cudaEvent_t *ev : {&hp->landed, &hp->computed, &hp->left})
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    if (e == cudaSuccess) {
      hp->link = &g_link[hp->device];
      if (take_link(*hp->link)) give_link(*hp->link);                // so that the first run does not wait for it
    }
  }
  if (e != cudaSuccess) {
    opencnn_host_plan_destroy(hp);
    return (int)e;
  }
  *plan = hp;
  return 0;
}

static int host_plan_async(void *plan, const float *input_host, const float *filter_host, float *output_host, bool kernels) {
  HostPlan *hp = static_cast<HostPlan *>(plan);
  if (!hp || !input_host || !filter_host || !output_host) return (int)cudaErrorInvalidValue;
  const size_t in_b = (size_t)hp->N * hp->C * hp->H * hp->W * 4, f_b = (size_t)hp->C * 9 * hp->K * 4;
  const size_t out_b = (size_t)hp->N * hp->K * hp->H * hp->W * 4;
  cudaError_t e = cudaMemcpyAsync(hp->d_filt, filter_host, f_b, cudaMemcpyHostToDevice, hp->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(hp->d_in, input_host, in_b, cudaMemcpyHostToDevice, hp->stream);
  if (e == cudaSuccess && kernels)
    e = forward(hp->d_in, hp->d_filt, hp->d_out, hp->d_ws, hp->N, hp->C, hp->H, hp->W, hp->K, hp->precision, hp->stream,
                shape_rule(hp->precision));
  if (e == cudaSuccess) e = cudaMemcpyAsync(output_host, hp->d_out, out_b, cudaMemcpyDeviceToHost, hp->stream);
  return (int)e;
}

int opencnn_host_plan_run_async(void *plan, const float *input_host, const float *filter_host,
                                float *output_host) {
  return host_plan_async(plan, input_host, filter_host, output_host, true);
}

int opencnn_host_plan_copy_async(void *plan, const float *input_host, const float *filter_host, float *output_host) {
  return host_plan_async(plan, input_host, filter_host, output_host, false);
}

int opencnn_host_plan_wait(void *plan) {
  HostPlan *hp = static_cast<HostPlan *>(plan);
  if (!hp) return (int)cudaErrorInvalidValue;
  return (int)cudaStreamSynchronize(hp->stream);
}

int opencnn_host_plan_run(void *plan, const float *input_host, const float *filter_host, float *output_host) {
  HostPlan *hp = static_cast<HostPlan *>(plan);
  if (!hp || !input_host || !filter_host || !output_host) return (int)cudaErrorInvalidValue;
  const size_t plane = (size_t)hp->N * hp->H * hp->W;
  int device = -1;
  const bool bands = hp->bands > 1 && bands_apart(input_host, hp->C * plane, output_host, hp->K * plane) && page_locked(input_host) &&
                     page_locked(output_host) && cudaGetDevice(&device) == cudaSuccess && device == hp->device &&
                     take_link(*hp->link);
  const cudaError_t e = bands ? run_bands(hp, input_host, filter_host, output_host)
                              : (cudaError_t)host_plan_async(plan, input_host, filter_host, output_host, true);
  // What was enqueued before an error still reads and writes the caller's memory: wait for it, too.  (run_bands may not have joined its streams.)
  cudaError_t w = cudaStreamSynchronize(hp->stream);
  if (bands) {
    if (e != cudaSuccess || w != cudaSuccess)
      for (cudaStream_t s : {hp->link->up, hp->link->down}) {
        const cudaError_t ws = cudaStreamSynchronize(s);
        if (w == cudaSuccess) w = ws;
      }
    give_link(*hp->link);
  }
  return (int)(e != cudaSuccess ? e : w);
}

int opencnn_host_plan_destroy(void *plan) {
  HostPlan *hp = static_cast<HostPlan *>(plan);
  if (!hp) return 0;
  for (cudaEvent_t ev : {hp->landed, hp->computed, hp->left})
    if (ev) cudaEventDestroy(ev);
  if (hp->d_in) cudaFree(hp->d_in);
  if (hp->d_filt) cudaFree(hp->d_filt);
  if (hp->d_out) cudaFree(hp->d_out);
  if (hp->d_ws) cudaFree(hp->d_ws);
  if (hp->stream) cudaStreamDestroy(hp->stream);
  delete hp;
  return 0;
}

}  // extern "C"
