// Arguments of the per-task entries, the mesh in the reference's numbering that
// they run on, and the permutations between that and the context's numbering.
#include "task_io.cuh"

namespace mpaso {

// Rows between the two numberings: dst[i] = src[perm[i]] or, SCATTER,
// dst[perm[i]] = src[i], a thread an element of V (two doubles where the row
// length and both addresses allow).
template <bool SCATTER, class V>
__global__ void __launch_bounds__(256) k_rows(const V *__restrict__ src, V *__restrict__ dst,
                                              const int32_t *__restrict__ perm, int64_t total, Lev row) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= total) return;
  int e, r;
  row.split(i, e, r);
  const int64_t j = (int64_t)perm[e] * row + r;
  if constexpr (SCATTER)
    dst[j] = src[i];
  else
    dst[i] = src[j];
}

namespace {
template <bool SCATTER>
void launch_rows(const double *src, double *dst, const int32_t *perm, int64_t n, int row, cudaStream_t s) {
  const int64_t total = n * row;
  if (row % 2 == 0 && (((uintptr_t)src | (uintptr_t)dst) & 15) == 0)
    k_rows<SCATTER><<<blocks_for(total / 2, 256), 256, 0, s>>>((const double2 *)src, (double2 *)dst, perm, total / 2,
                                                               row / 2);
  else
    k_rows<SCATTER><<<blocks_for(total, 256), 256, 0, s>>>(src, dst, perm, total, row);
  MPASO_CUDA(cudaGetLastError());
}
}  // namespace

// Rows between page-locked host memory (reference order, read or written
// through its device alias) and device memory (context order), in one pass:
// the host side is walked in order, 16 bytes a thread where both sides allow
// (coalesced over the host link), and the device side is scattered through
// iperm (reference id -> context id).  import: dst[iperm[j]] = src[j];
// export: dst[j] = src[iperm[j]] (rows of `row` doubles).
template <bool IMPORT>
__global__ void k_host_rows(const double *__restrict__ src, double *__restrict__ dst,
                            const int32_t *__restrict__ iperm, int64_t n, Lev row, bool pairs) {
  const int64_t total = n * row, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  auto dev = [&](int64_t i) {
    int j, r;
    row.split(i, j, r);
    return (int64_t)iperm[j] * row + r;
  };
  if (pairs) {  // total even, host side 16-byte aligned
    for (int64_t p = t0; p < total / 2; p += stride) {
      const int64_t i = 2 * p;
      if constexpr (IMPORT) {
        const double2 v = reinterpret_cast<const double2 *>(src)[p];
        dst[dev(i)] = v.x;
        dst[dev(i + 1)] = v.y;
      } else {
        reinterpret_cast<double2 *>(dst)[p] = make_double2(src[dev(i)], src[dev(i + 1)]);
      }
    }
  } else {
    for (int64_t i = t0; i < total; i += stride) {
      if constexpr (IMPORT)
        dst[dev(i)] = src[i];
      else
        dst[i] = src[dev(i)];
    }
  }
}

void host_rows_pub(bool import, const double *src, double *dst, const int32_t *iperm, int64_t n, int row,
                   int sms, cudaStream_t s) {
  const int64_t total = n * row;
  const double *host = import ? src : dst;
  const bool pairs = total % 2 == 0 && ((uintptr_t)host & 15) == 0;
  const int64_t work = pairs ? total / 2 : total;
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(blocks_for(work, 256), (int64_t)sms * 8));
  if (import)
    k_host_rows<true><<<blocks, 256, 0, s>>>(src, dst, iperm, n, row, pairs);
  else
    k_host_rows<false><<<blocks, 256, 0, s>>>(src, dst, iperm, n, row, pairs);
  MPASO_CUDA(cudaGetLastError());
}

void k_gather_rows_pub(const double *src, double *dst, const int32_t *perm, int64_t n, int row,
                       cudaStream_t s) {
  launch_rows<false>(src, dst, perm, n, row, s);
}

void k_scatter_rows_pub(const double *src, double *dst, const int32_t *perm, int64_t n, int row,
                        cudaStream_t s) {
  launch_rows<true>(src, dst, perm, n, row, s);
}

bool is_device_pointer(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

TaskIO::TaskIO(mpaso_mesh m, void *stream) : m_(m) {
  require(m != nullptr, MPASO_ERR_ARG, "null mesh context");
  MPASO_CUDA(cudaSetDevice(m->ctx.device));
  stream_ = stream ? (cudaStream_t)stream : m->ctx.stream;
}

TaskIO::~TaskIO() = default;

int64_t TaskIO::count(int entity) const {
  const DMesh &d = m_->ctx.d;
  return entity == MPASO_CELLS ? d.nC : entity == MPASO_EDGES ? d.nE : d.nV;
}

int TaskIO::add(const double *p, int entity, int row, bool output) {
  require(p != nullptr, MPASO_ERR_ARG, "null field pointer");
  require(row >= 1, MPASO_ERR_ARG, "bad row length");
  Arg a{const_cast<double *>(p), entity, row, output, !is_device_pointer(p)};
  any_host_ |= a.host;
  args_.push_back(a);
  return (int)args_.size() - 1;
}

// Whether an output shares memory with another argument: the kernels then
// work on copies, so that every input is read as it was before the call.
bool TaskIO::overlapping() const {
  for (size_t x = 0; x < args_.size(); ++x) {
    if (!args_[x].output) continue;
    const double *x0 = args_[x].user, *x1 = x0 + count(args_[x].entity) * args_[x].row;
    for (size_t y = 0; y < args_.size(); ++y) {
      const double *y0 = args_[y].user, *y1 = y0 + count(args_[y].entity) * args_[y].row;
      if (x != y && x0 < y1 && y0 < x1) return true;
    }
  }
  return false;
}

void TaskIO::stage() {
  m_->ctx.task_view();
  copies_ = overlapping();
  size_t total = 0;
  auto bytes_of = [&](const Arg &a) { return (size_t)count(a.entity) * a.row * sizeof(double); };
  for (auto &a : args_)
    if (a.host || copies_) total += (bytes_of(a) + 255) & ~size_t(255);
  char *base = total ? (char *)m_->ctx.ensure_scratch(total) : nullptr;
  for (auto &a : args_) {
    if (!a.host && !copies_) {
      a.internal = a.user;
      continue;
    }
    a.internal = (double *)base;
    base += (bytes_of(a) + 255) & ~size_t(255);
    MPASO_CUDA(cudaMemcpyAsync(a.internal, a.user, bytes_of(a),
                               a.host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, stream_));
  }
}

void TaskIO::finish() {
  MPASO_CUDA(cudaGetLastError());
  for (auto &a : args_)
    if (a.output && (a.host || copies_))
      MPASO_CUDA(cudaMemcpyAsync(a.user, a.internal, (size_t)count(a.entity) * a.row * sizeof(double),
                                 a.host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, stream_));
  if (any_host_) MPASO_CUDA(cudaStreamSynchronize(stream_));
}

// ------------------------------------------- the mesh in the reference's numbering
//
// Permuting every argument into the context's numbering and back cost two
// launches and two passes a field (57 launches for a task-by-task ocean tracer
// stage; level 5, 20 levels x 3 tracers: 573 us, in the view 456 us), more than
// the curve order saves a task that reads each field once.
namespace {

__device__ __forceinline__ int ref_id(int v, const int32_t *to_ref) { return to_ref ? to_ref[v] : v; }
__device__ __forceinline__ double ref_id(double v, const int32_t *) { return v; }
__device__ __forceinline__ int2 ref_id(int2 v, const int32_t *to_ref) {
  return make_int2(to_ref[v.x], to_ref[v.y]);
}

// A slot-major [slots][n] array (or, by_row, an [n][slots] one) from the
// context's numbering into the reference's; the ids it holds (to_ref given)
// change with it.
template <class T>
__global__ void k_to_reference(const T *__restrict__ src, T *__restrict__ dst, const int32_t *__restrict__ to_ctx,
                               const int32_t *__restrict__ to_ref, int64_t n, int slots, bool by_row) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * slots) return;
  const int64_t r = by_row ? i / slots : i % n, j = by_row ? i % slots : i / n;
  const int64_t c = to_ctx[r];
  dst[i] = ref_id(src[by_row ? c * slots + j : j * n + c], to_ref);
}

}  // namespace

// Built on a stream of its own with the thread's capture mode relaxed: the
// call that needs it first may be recorded into a graph, and the view must
// exist before that graph is launched.
const DMesh &MeshCtx::task_view() {
  std::lock_guard<std::mutex> lock(ref_mutex);
  if (has_ref) return ref;
  bool same = true;
  for (const auto &p : perm)
    for (size_t i = 0; i < p.size() && same; ++i) same = p[i] == (int32_t)i;
  if (same) {
    ref = d, has_ref = true;
    return ref;
  }
  DMesh m = d;
  struct Item {
    void *pp;  // the pointer of `m` to replace
    int kind;  // bytes per element
    int entity, slots, ids;
    bool by_row;
  };
  const int E = std::max(d.maxEoE, 1);
  const Item items[] = {
      {&m.nEoC, 4, MPASO_CELLS, 1, -1, false}, {&m.eoc, 4, MPASO_CELLS, d.maxEoC, MPASO_EDGES, false},
      {&m.eocSign, 8, MPASO_CELLS, d.maxEoC, -1, false}, {&m.eocAsc, 4, MPASO_CELLS, d.maxEoC, MPASO_EDGES, false},
      {&m.eocAscSign, 8, MPASO_CELLS, d.maxEoC, -1, false}, {&m.coc, 4, MPASO_CELLS, d.maxEoC, MPASO_CELLS, false},
      {&m.areaCell, 8, MPASO_CELLS, 1, -1, false}, {&m.invAreaCell, 8, MPASO_CELLS, 1, -1, false},
      {&m.bottomDepth, 8, MPASO_CELLS, 1, -1, false}, {&m.maxLevelCell, 4, MPASO_CELLS, 1, -1, false},
      {&m.coe, 16, MPASO_EDGES, 1, MPASO_CELLS, false}, {&m.voe, 16, MPASO_EDGES, 1, MPASO_VERTICES, false},
      {&m.dvEdge, 8, MPASO_EDGES, 1, -1, false}, {&m.dcEdge, 8, MPASO_EDGES, 1, -1, false},
      {&m.nEoE, 4, MPASO_EDGES, 1, -1, false}, {&m.eoe, 4, MPASO_EDGES, E, MPASO_EDGES, false},
      {&m.woe, 8, MPASO_EDGES, E, -1, false}, {&m.maxLevelEdgeTop, 4, MPASO_EDGES, 1, -1, false},
      {&m.nAdv, 4, MPASO_EDGES, 1, -1, false}, {&m.advCells, 4, MPASO_EDGES, d.maxAdv, MPASO_CELLS, false},
      {&m.advCp, 8, MPASO_EDGES, d.maxAdv, -1, false}, {&m.advCm, 8, MPASO_EDGES, d.maxAdv, -1, false},
      {&m.hoMask, 4, MPASO_EDGES, d.fctLev, -1, true}, {&m.meshScalingDel2, 8, MPASO_EDGES, 1, -1, false},
      {&m.cov, 4, MPASO_VERTICES, kVertexDegree, MPASO_CELLS, false},
      {&m.kite, 8, MPASO_VERTICES, kVertexDegree, -1, false},
      {&m.eov, 4, MPASO_VERTICES, kVertexDegree, MPASO_EDGES, false},
      {&m.eovSign, 8, MPASO_VERTICES, kVertexDegree, -1, false},
      {&m.areaTriangle, 8, MPASO_VERTICES, 1, -1, false}, {&m.fVertex, 8, MPASO_VERTICES, 1, -1, false}};
  const int64_t cnt[3] = {d.nC, d.nE, d.nV};
  auto bytes_of = [&](const Item &t) {
    return ((size_t)cnt[t.entity] * t.slots * (t.kind == 16 ? 8 : t.kind) + 255) & ~size_t(255);
  };
  size_t total = 0;
  for (const Item &t : items) total += bytes_of(t);
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaStream_t stream = nullptr;
    Relaxed() { MPASO_CUDA(cudaThreadExchangeStreamCaptureMode(&mode)); }
    ~Relaxed() {
      if (stream) cudaStreamDestroy(stream);
      cudaThreadExchangeStreamCaptureMode(&mode);
    }
  } own;
  MPASO_CUDA(cudaStreamCreateWithFlags(&own.stream, cudaStreamNonBlocking));
  const cudaStream_t stream = own.stream;
  void *arena_new = nullptr;
  if (cudaMalloc(&arena_new, total) != cudaSuccess) {
    cudaGetLastError();
    fail(MPASO_ERR_ALLOC, "device allocation of the task view failed (" + std::to_string(total) + " bytes)");
  }
  try {
    char *base = (char *)arena_new;
    for (const Item &t : items) {
      const int64_t n = cnt[t.entity];
      const int32_t *to_ctx = d_iperm[t.entity], *to_ref = t.ids < 0 ? nullptr : d_perm[t.ids];
      const int b = blocks_for(n * t.slots, 256);
      const void *src = *(const void **)t.pp;
      if (t.kind == 4)
        k_to_reference<<<b, 256, 0, stream>>>((const int *)src, (int *)base, to_ctx, to_ref, n, t.slots, t.by_row);
      else if (t.kind == 8)
        k_to_reference<<<b, 256, 0, stream>>>((const double *)src, (double *)base, to_ctx, to_ref, n, t.slots, t.by_row);
      else
        k_to_reference<<<b, 256, 0, stream>>>((const int2 *)src, (int2 *)base, to_ctx, to_ref, n, t.slots, t.by_row);
      *(const void **)t.pp = base;
      base += bytes_of(t);
    }
    MPASO_CUDA(cudaGetLastError());
    MPASO_CUDA(cudaStreamSynchronize(stream));  // any stream may use it from here on
  } catch (...) {
    cudaFree(arena_new);
    throw;
  }
  // what no task kernel reads keeps no pointer into the other numbering
  m.nbr = nullptr, m.invDcEdge = m.invDvEdge = nullptr, m.advCoef = m.advCoef3 = nullptr, m.invAreaTriangle = nullptr;
  m.woeT = m.kiteR = nullptr, m.vocR = m.advRe = m.cocU = nullptr, m.advRc = nullptr;
  ref = m, ref_arena = arena_new, ref_bytes = total, has_ref = true;
  return ref;
}

}  // namespace mpaso
