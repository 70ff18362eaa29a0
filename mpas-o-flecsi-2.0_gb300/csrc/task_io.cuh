// Arguments of the per-task entries.  The task kernels run in the reference's
// numbering (MeshCtx::task_view) on device arrays where they lie; host arrays
// are copied in and back out.
#pragma once

#include "device.cuh"

namespace mpaso {

bool is_device_pointer(const void *p);
// One pass between a page-locked host array (reference order, through its
// device alias) and a device array (context order): import (host -> device)
// or export; iperm maps reference ids to context ids.
void host_rows_pub(bool import, const double *src, double *dst, const int32_t *iperm, int64_t n, int row,
                   int sms, cudaStream_t s);
void k_gather_rows_pub(const double *src, double *dst, const int32_t *perm, int64_t n, int row,
                       cudaStream_t s);
void k_scatter_rows_pub(const double *src, double *dst, const int32_t *perm, int64_t n, int row,
                        cudaStream_t s);

class TaskIO {
 public:
  TaskIO(mpaso_mesh m, void *stream);
  ~TaskIO();
  // Registers an argument; returns its slot.  `entity` = MPASO_CELLS/EDGES/VERTICES,
  // `row` = doubles per entity.  Entries of an output that a task leaves untouched
  // keep their values (FleCSI storage semantics): staged outputs are copied in as well.
  int in(const double *p, int entity, int row) { return add(p, entity, row, false); }
  int out(double *p, int entity, int row) { return add(p, entity, row, true); }
  void stage();                  // copies host arrays in
  double *ptr(int slot) const { return args_[slot].internal; }
  void finish();                 // copies outputs back, syncs for host memory
  cudaStream_t stream() const { return stream_; }
  MeshCtx &ctx() { return m_->ctx; }
  const DMesh &dm() const { return m_->ctx.ref; }  // reference numbering, valid after stage()

 private:
  struct Arg {
    double *user;
    int entity, row;
    bool output, host;
    double *internal = nullptr;
  };
  int add(const double *p, int entity, int row, bool output);
  int64_t count(int entity) const;
  bool overlapping() const;
  mpaso_mesh m_;
  cudaStream_t stream_;
  std::vector<Arg> args_;
  bool any_host_ = false, copies_ = false;
};

}  // namespace mpaso
