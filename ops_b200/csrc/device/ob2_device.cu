// ob2_device.cu -- CUDA side of the thin C ABI (include/ops_b200_device.h):
// device selection, the work stream, memory, events, halo transfer, box
// copies and fills.  Kernels here are HBM-bound byte/element moves: no tensor
// cores; coalesced along x, grids sized from the SM count.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>

#include "ops_b200_device.h"

namespace {

// CUDA's lazy module loading (the default since CUDA 12.2) loads a kernel at
// its first launch; in a process that alternates kernels of several
// libraries (an application's generated kernels, then this library's), a
// launch of this library's x-direction tridiagonal kernel blocked about
// 220 us on the host at every ADI step with the device left idle meanwhile
// (256^3 FP64 ADI step: 1.13 ms lazy, 0.89 ms eager, measured).  So when
// the library is loaded, before any CUDA call of the process, it asks for
// eager loading unless the process chose a mode itself (an explicit
// CUDA_MODULE_LOADING=LAZY is kept).  A process that initialised CUDA
// before loading the library keeps the mode it started with.
__attribute__((constructor)) void ob2_module_loading() {
  if (!getenv("CUDA_MODULE_LOADING")) setenv("CUDA_MODULE_LOADING", "EAGER", 0);
}

cudaStream_t g_stream = nullptr;   // current work stream
cudaStream_t g_default = nullptr;  // the runtime's own non-blocking stream
int g_sms = 148;
int g_device = -1;                 // the device ob2_dev_init selected

inline int rc(cudaError_t e) { return (int)e; }

}  // namespace

OB2_API int ob2_dev_init(int device) {
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess) return rc(e);
  if (n == 0) return (int)cudaErrorNoDevice;
  if (device < 0 || device >= n) device = 0;
  e = cudaSetDevice(device);
  if (e != cudaSuccess) return rc(e);
  g_device = device;
  cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, device);
  if (!g_default) {
    e = cudaStreamCreateWithFlags(&g_default, cudaStreamNonBlocking);
    if (e != cudaSuccess) return rc(e);
  }
  g_stream = g_default;
  return 0;
}

OB2_API int ob2_dev_count(int *n) { return rc(cudaGetDeviceCount(n)); }
OB2_API int ob2_dev_sm_count(int *n) {
  *n = g_sms;
  return 0;
}
OB2_API void *ob2_dev_stream(void) { return (void *)g_stream; }
OB2_API int ob2_dev_set_stream(void *s) {
  g_stream = s ? (cudaStream_t)s : g_default;
  return 0;
}
OB2_API int ob2_dev_malloc(void **p, size_t n) { return rc(cudaMalloc(p, n ? n : 16)); }
OB2_API int ob2_dev_free(void *p) { return p ? rc(cudaFree(p)) : 0; }
OB2_API int ob2_dev_memset(void *p, int v, size_t n) {
  return rc(cudaMemsetAsync(p, v, n, g_stream));
}
OB2_API int ob2_dev_h2d(void *dst, const void *src, size_t n) {
  cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, g_stream);
  if (e != cudaSuccess) return rc(e);
  return rc(cudaStreamSynchronize(g_stream));
}
OB2_API int ob2_dev_d2h(void *dst, const void *src, size_t n) {
  cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, g_stream);
  if (e != cudaSuccess) return rc(e);
  return rc(cudaStreamSynchronize(g_stream));
}
OB2_API int ob2_dev_d2d(void *dst, const void *src, size_t n) {
  return rc(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToDevice, g_stream));
}
OB2_API int ob2_dev_h2d_async(void *dst, const void *src, size_t n) {
  return rc(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, g_stream));
}
OB2_API int ob2_dev_d2h_async(void *dst, const void *src, size_t n) {
  return rc(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, g_stream));
}
OB2_API int ob2_dev_sync(void) { return rc(cudaStreamSynchronize(g_stream)); }
OB2_API int ob2_host_alloc_pinned(void **p, size_t n) {
  return rc(cudaHostAlloc(p, n ? n : 16, cudaHostAllocPortable));
}
OB2_API int ob2_host_free_pinned(void *p) { return p ? rc(cudaFreeHost(p)) : 0; }
OB2_API const char *ob2_error_string(int code) {
  if (code == OB2_ERR_NOALLOC_LIMIT)
    return "halo task table larger than the allocation-free maximum (OB2_HALO_STATIC_MAX)";
  return cudaGetErrorString((cudaError_t)code);
}
OB2_API int ob2_last_launch_error(void) { return rc(cudaGetLastError()); }
OB2_API int ob2_mem_info(size_t *f, size_t *t) { return rc(cudaMemGetInfo(f, t)); }

OB2_API int ob2_event_create(void **ev) {
  return rc(cudaEventCreate((cudaEvent_t *)ev));
}
OB2_API int ob2_event_record(void *ev) { return rc(cudaEventRecord((cudaEvent_t)ev, g_stream)); }
OB2_API int ob2_event_elapsed_ms(void *a, void *b, float *ms) {
  cudaError_t e = cudaEventSynchronize((cudaEvent_t)b);
  if (e != cudaSuccess) return rc(e);
  return rc(cudaEventElapsedTime(ms, (cudaEvent_t)a, (cudaEvent_t)b));
}
OB2_API int ob2_event_destroy(void *ev) { return rc(cudaEventDestroy((cudaEvent_t)ev)); }

// ---------------------------------------------------------------------------
// Halo transfer: one CTA row (blockIdx.y) per halo task, threads stride over
// the task's points.  Index math mirrors the oracle restatement of
// ops_host_singlenode.cpp:172-446: iteration point t -> per-dimension storage
// index start + (flip ? L-1-t_axis : t_axis).
// ---------------------------------------------------------------------------
namespace {

// element offset (points) of iteration point t of a box of extents n in a dat
__device__ __forceinline__ long long storage_offset(const int *axis, const int *flip,
                                                    const int *start, const long long *cum,
                                                    const int (&t)[3], const int (&n)[3]) {
  long long off = 0;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const int a = axis[i];  // selected, not indexed: t and n stay in registers
    const int ta = a == 0 ? t[0] : a == 1 ? t[1] : t[2];
    const int na = a == 0 ? n[0] : a == 1 ? n[1] : n[2];
    off += (long long)(start[i] + (flip[i] ? na - 1 - ta : ta)) * cum[i];
  }
  return off;
}

__device__ __forceinline__ double load_as_double(const char *p, int ts) {
  if (ts == 8) return *(const double *)p;
  if (ts == 2) return (double)__half2float(*(const __half *)p);
  return (double)*(const float *)p;
}

__global__ void halo_kernel(const ob2_halo_task *__restrict__ tasks) {
  const ob2_halo_task &T = tasks[blockIdx.y];
  const int n[3] = {T.iter[0], T.iter[1], T.iter[2]};
  const bool small = T.npts >> 31 == 0;  // 32-bit division
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < T.npts;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = small ? (long long)((unsigned)i / (unsigned)n[0]) : i / n[0];
    const long long z = small ? (long long)((unsigned)r / (unsigned)n[1]) : r / n[1];
    const int t[3] = {(int)(i - r * n[0]), (int)(r - z * n[1]), (int)z};
    const long long so = storage_offset(T.src_axis, T.src_flip, T.src_start, T.src_cum, t, n);
    const long long dof = storage_offset(T.dst_axis, T.dst_flip, T.dst_start, T.dst_cum, t, n);
    for (int c = 0; c < T.ncomp; c++) {
      long long se = T.src_soa ? so + c * T.src_npts_total : so * T.ncomp + c;
      long long de = T.dst_soa ? dof + c * T.dst_npts_total : dof * T.ncomp + c;
      const char *sp = T.src + se * T.src_type;
      char *dp = T.dst + de * T.dst_type;
      if (T.src_type == T.dst_type) {
        if (T.src_type == 8)
          *(unsigned long long *)dp = *(const unsigned long long *)sp;
        else if (T.src_type == 4)
          *(unsigned int *)dp = *(const unsigned int *)sp;
        else if (T.src_type == 2)
          *(unsigned short *)dp = *(const unsigned short *)sp;
        else
          for (int b = 0; b < T.src_type; b++) dp[b] = sp[b];
      } else {
        double v = load_as_double(sp, T.src_type);
        if (T.dst_type == 8)
          *(double *)dp = v;
        else if (T.dst_type == 2)
          *(__half *)dp = __double2half(v);
        else
          *(float *)dp = (float)v;
      }
    }
  }
}

}  // namespace

OB2_API int ob2_halo_run(const ob2_halo_task *tasks_dev, int ntasks, long long max_pts) {
  if (ntasks <= 0 || max_pts <= 0) return 0;
  long long blocks = (max_pts + 255) / 256;
  if (blocks > 4LL * g_sms) blocks = 4LL * g_sms;
  dim3 grid((unsigned)blocks, (unsigned)ntasks);
  halo_kernel<<<grid, 256, 0, g_stream>>>(tasks_dev);
  return rc(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Allocation-free halo transfer: the task table lives in a fixed array
// compiled into this library instead of caller-allocated device memory.
// ---------------------------------------------------------------------------
namespace {

__device__ __align__(256) ob2_halo_task g_halo_static[OB2_HALO_STATIC_MAX];

constexpr int kMaxDevices = 64;
// device address of g_halo_static, looked up once per device (host code may
// not pass the symbol itself to a kernel: its host-side name is a stand-in);
// atomic so that first calls from several host threads do not race
std::atomic<ob2_halo_task *> g_halo_static_addr[kMaxDevices];

}  // namespace

OB2_API int ob2_halo_run_noalloc(const ob2_halo_task *tasks_host, int ntasks) {
  if (ntasks < 0 || (ntasks > 0 && !tasks_host)) return (int)cudaErrorInvalidValue;
  if (ntasks > OB2_HALO_STATIC_MAX) return OB2_ERR_NOALLOC_LIMIT;
  if (ntasks == 0) return 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return rc(e);
  if (dev < 0 || dev >= kMaxDevices) return (int)cudaErrorInvalidDevice;
  // the launch goes to the work stream, which belongs to the device that
  // ob2_dev_init selected: the array looked up must be that device's
  if (g_device >= 0 && dev != g_device) return (int)cudaErrorInvalidDevice;
  ob2_halo_task *table = g_halo_static_addr[dev].load(std::memory_order_acquire);
  if (!table) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_halo_static);
    if (e != cudaSuccess) return rc(e);
    table = (ob2_halo_task *)p;
    g_halo_static_addr[dev].store(table, std::memory_order_release);
  }
  long long max_pts = 0;
  for (int i = 0; i < ntasks; i++)
    if (tasks_host[i].npts > max_pts) max_pts = tasks_host[i].npts;
  // stream-ordered: an earlier launch on this stream still reading the table
  // finishes before it is overwritten
  e = cudaMemcpyAsync(table, tasks_host, sizeof(ob2_halo_task) * ntasks,
                      cudaMemcpyHostToDevice, g_stream);
  if (e != cudaSuccess) return rc(e);
  return ob2_halo_run(table, ntasks, max_pts);
}

// ---------------------------------------------------------------------------
// Box copy between a dat (storage coordinates start3/count3) and a dense AoS
// buffer, for fetch/set data and slabs (ops_util.cpp:353-500 semantics).
//
// Bound by HBM: one read and one write per element.  A row of the box is
// c0 * nc elements, contiguous in the buffer and in an AoS dat, so a group of
// LR lanes (the smallest power of two that covers a row, at most a warp)
// copies a row, or a piece of kPiece units of a long one, with four accesses
// per lane in flight and one division per row; a 187 x 180 x 139 box of 3
// FP64 components (112 MB each way) takes 39 us against 64 us for one
// element per thread with two 64-bit divisions and a component loop.
// Components of a SoA dat lie apart (SOA): the lanes take the units of the
// buffer's row in turn, each from its component's own row in the dat.
// ---------------------------------------------------------------------------
namespace {

constexpr int kPiece = 1024;  // units of a row that one group copies at a time

struct BoxRows {
  long long off, pitch, plane;  // first unit of the box in the dat; per row; per plane
  long long len, bstep;         // units per row, buffer units per row
  long long rows;               // c1 * c2
  int c1, npiece, lr;           // rows per plane, pieces per row, log2 lanes
  int w, per;                   // SOA: units of an element, of a point in the buffer
  long long comp;               // SOA: units from one component to the next in the dat
  int dir;                      // 0 dat -> buffer, 1 buffer -> dat
};

template <typename U, bool SOA>
__global__ void __launch_bounds__(256) box_copy_kernel(U *__restrict__ dat, U *__restrict__ buf,
                                                       const BoxRows g) {
  const int lane = threadIdx.x & ((1 << g.lr) - 1), ln = 1 << g.lr;
  const long long items = g.rows * g.npiece;
  const long long step = (long long)gridDim.x * (blockDim.x >> g.lr);
  const int sx = SOA ? ln / g.per : 0, sk = SOA ? ln % g.per : 0;  // ln units on
  for (long long it = (long long)blockIdx.x * (blockDim.x >> g.lr) + (threadIdx.x >> g.lr);
       it < items; it += step) {
    long long row = it, z;
    int piece = 0;
    if (g.npiece > 1) {
      row = it / g.npiece;
      piece = (int)(it - row * g.npiece);
    }
    if (g.rows >> 31)
      z = row / g.c1;
    else
      z = (int)row / g.c1;
    const int y = (int)(row - z * g.c1);
    U *d = dat + g.off + z * g.plane + y * g.pitch;
    U *b = buf + row * g.bstep;
    const long long end = g.npiece > 1 ? min(g.len, (long long)(piece + 1) * kPiece) : g.len;
    long long e = (long long)piece * kPiece + lane;
    // SOA: unit e of the row is unit k of point x
    long long x = SOA ? (g.len >> 31 ? e / g.per : (long long)((unsigned)e / (unsigned)g.per)) : 0;
    int k = SOA ? (int)(e - x * g.per) : 0;
    // where unit e + j * ln lies in the dat's row (asked for in order)
    auto at = [&](int j) {
      if (!SOA) return e + j * ln;
      const long long o = g.w == 1 ? x + k * g.comp : x * g.w + k / g.w * g.comp + k % g.w;
      x += sx;
      k += sk;
      if (k >= g.per) {
        k -= g.per;
        x++;
      }
      return o;
    };
    U v[4];
    if (g.dir == 0) {
      for (; e + 3 * ln < end; e += 4 * ln) {
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = d[at(j)];
#pragma unroll
        for (int j = 0; j < 4; j++) b[e + j * ln] = v[j];
      }
      for (; e < end; e += ln) b[e] = d[at(0)];
    } else {
      for (; e + 3 * ln < end; e += 4 * ln) {
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = b[e + j * ln];
#pragma unroll
        for (int j = 0; j < 4; j++) d[at(j)] = v[j];
      }
      for (; e < end; e += ln) d[at(0)] = b[e];
    }
  }
}

template <typename U>
int launch_box(char *dat, char *buf, BoxRows g, bool apart) {
  g.lr = 0;
  while (g.lr < 5 && (1LL << g.lr) < g.len) g.lr++;
  g.npiece = (int)((g.len + kPiece - 1) / kPiece);
  const long long per = 256 >> g.lr;
  const long long need = (g.rows * g.npiece + per - 1) / per;
  const unsigned blocks = (unsigned)std::min(need, 32LL * g_sms);
  if (apart)
    box_copy_kernel<U, true><<<blocks, 256, 0, g_stream>>>((U *)dat, (U *)buf, g);
  else
    box_copy_kernel<U, false><<<blocks, 256, 0, g_stream>>>((U *)dat, (U *)buf, g);
  return rc(cudaGetLastError());
}

}  // namespace

OB2_API int ob2_box_copy(char *dat, int ts, int nc, int soa, const int *size3, const int *start3,
                         const int *count3, char *buf, int dir) {
  if ((long long)count3[0] * count3[1] * count3[2] <= 0 || nc <= 0 || ts <= 0) return 0;
  // copied in units of 8, 4, 2 or 1 bytes: the widest that divides the
  // element and both addresses
  int u = 8;
  while (u > 1 && ((uintptr_t)dat % u || (uintptr_t)buf % u || ts % u)) u >>= 1;
  const int w = ts / u;  // units per element
  const long long sx = size3[0], sy = (long long)size3[0] * size3[1];
  const long long pt = start3[0] + start3[1] * sx + start3[2] * sy;
  const bool apart = soa && nc > 1;
  const long long m = apart ? w : (long long)nc * w;  // units per point in the dat
  BoxRows g;
  g.off = pt * m;
  g.pitch = sx * m;
  g.plane = sy * m;
  g.rows = (long long)count3[1] * count3[2];
  g.bstep = (long long)count3[0] * nc * w;
  g.c1 = count3[1];
  g.dir = dir;
  g.len = g.bstep;
  g.w = w;
  g.per = nc * w;
  g.comp = sy * size3[2] * w;
  return u == 8   ? launch_box<unsigned long long>(dat, buf, g, apart)
         : u == 4 ? launch_box<unsigned int>(dat, buf, g, apart)
         : u == 2 ? launch_box<unsigned short>(dat, buf, g, apart)
                  : launch_box<unsigned char>(dat, buf, g, apart);
}

// ---------------------------------------------------------------------------
// Fills
// ---------------------------------------------------------------------------
namespace {

__global__ void fill_kernel(char *p, unsigned long long v, int ts, size_t count) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (size_t)gridDim.x * blockDim.x) {
    if (ts == 8)
      ((unsigned long long *)p)[i] = v;
    else if (ts == 4)
      ((unsigned int *)p)[i] = (unsigned int)v;
    else if (ts == 2)
      ((unsigned short *)p)[i] = (unsigned short)v;
    else
      p[i] = (char)v;
  }
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

__global__ void random_kernel(char *p, int ts, size_t count, unsigned long long seed,
                              unsigned long long counter, int normal) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (size_t)gridDim.x * blockDim.x) {
    unsigned long long k = counter + i;
    unsigned long long r1 = mix64(seed * 0x100000001b3ULL ^ (2 * k));
    double u1 = (double)(r1 >> 11) * (1.0 / 9007199254740992.0);
    double v = u1;
    if (normal) {
      unsigned long long r2 = mix64(seed * 0x100000001b3ULL ^ (2 * k + 1));
      double u2 = (double)(r2 >> 11) * (1.0 / 9007199254740992.0);
      v = sqrt(-2.0 * log(1.0 - u1)) * cos(6.283185307179586 * u2);
    }
    if (ts == 8)
      ((double *)p)[i] = v;
    else
      ((float *)p)[i] = (float)v;
  }
}

}  // namespace

namespace {
template <typename T>
__global__ void nan_find_kernel(const T *__restrict__ p, int ncomp, int soa, size_t count,
                                unsigned long long *first) {
  const size_t npts = count / (size_t)ncomp;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count;
       e += (size_t)gridDim.x * blockDim.x) {
    const T v = p[e];
    if (v != v) {
      const unsigned long long key =
          soa ? (unsigned long long)(e % npts) * ncomp + e / npts : (unsigned long long)e;
      atomicMin(first, key);
    }
  }
}
}  // namespace

OB2_API int ob2_nan_find(const void *p, int ts, int ncomp, int soa, size_t count,
                         long long *first) {
  *first = -1;
  if (count == 0 || ncomp < 1) return 0;
  if (ts != 8 && ts != 4) return (int)cudaErrorInvalidValue;
  unsigned long long *d = nullptr, h = ~0ULL;
  cudaError_t e = cudaMallocAsync(&d, sizeof(h), g_stream);
  if (e != cudaSuccess) return rc(e);
  e = cudaMemcpyAsync(d, &h, sizeof(h), cudaMemcpyHostToDevice, g_stream);
  const unsigned blocks = (unsigned)std::min<size_t>((count + 255) / 256, (size_t)g_sms * 8);
  if (e == cudaSuccess) {
    if (ts == 8)
      nan_find_kernel<double><<<blocks, 256, 0, g_stream>>>((const double *)p, ncomp, soa, count, d);
    else
      nan_find_kernel<float><<<blocks, 256, 0, g_stream>>>((const float *)p, ncomp, soa, count, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, g_stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g_stream);
  cudaFreeAsync(d, g_stream);
  if (e != cudaSuccess) return rc(e);
  *first = h == ~0ULL ? -1 : (long long)h;
  return 0;
}

OB2_API int ob2_fill_value(void *p, const void *val, int ts, size_t count) {
  if (count == 0) return 0;
  if (ts == 16) {  // a complex value whose two halves are equal: 2 count 8-byte values
    if (memcmp(val, (const char *)val + 8, 8) != 0) return (int)cudaErrorInvalidValue;
    ts = 8;
    count *= 2;
  }
  if (ts > 8 || ts < 1) return (int)cudaErrorInvalidValue;
  unsigned long long v = 0;
  memcpy(&v, val, ts <= 8 ? ts : 8);
  size_t blocks = (count + 255) / 256;
  if (blocks > (size_t)8 * g_sms) blocks = (size_t)8 * g_sms;
  fill_kernel<<<(unsigned)blocks, 256, 0, g_stream>>>((char *)p, v, ts, count);
  return rc(cudaGetLastError());
}

OB2_API int ob2_fill_random(void *p, int ts, size_t count, unsigned long long seed,
                            unsigned long long counter, int normal) {
  if (count == 0) return 0;
  size_t blocks = (count + 255) / 256;
  if (blocks > (size_t)8 * g_sms) blocks = (size_t)8 * g_sms;
  random_kernel<<<(unsigned)blocks, 256, 0, g_stream>>>((char *)p, ts, count, seed, counter,
                                                          normal);
  return rc(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Graph capture of the work stream (loop chains)
// ---------------------------------------------------------------------------
OB2_API int ob2_graph_begin_capture(void) {
  return rc(cudaStreamBeginCapture(g_stream, cudaStreamCaptureModeThreadLocal));
}
OB2_API int ob2_graph_end_capture(void **exec) {
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamEndCapture(g_stream, &g);
  if (e != cudaSuccess) return rc(e);
  if (*exec) {
    cudaGraphExecUpdateResultInfo info;
    e = cudaGraphExecUpdate((cudaGraphExec_t)*exec, g, &info);
    if (e == cudaSuccess) {
      cudaGraphDestroy(g);
      return 0;
    }
    (void)cudaGetLastError();  // a refused update is not an error
    cudaGraphExecDestroy((cudaGraphExec_t)*exec);
    *exec = nullptr;
  }
  cudaGraphExec_t ge = nullptr;
  e = cudaGraphInstantiate(&ge, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return rc(e);
  *exec = (void *)ge;
  return 0;
}
OB2_API int ob2_graph_launch(void *exec) {
  return rc(cudaGraphLaunch((cudaGraphExec_t)exec, g_stream));
}
OB2_API int ob2_graph_destroy(void *exec) {
  return exec ? rc(cudaGraphExecDestroy((cudaGraphExec_t)exec)) : 0;
}
