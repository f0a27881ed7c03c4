// Moves the interface tensors of a program between the caller's host buffers and the device.
//
// What bounds it: a small transfer is all latency (a copy-engine copy costs about 5 us of host and
// device time, and one per tensor adds up to the length of a small model's pass).  So tensors of at most
// kSmall bytes go through a page-locked image that a kernel reads or writes
// directly, neighbours in one launch (a two-layer encoder at 16 tokens: 195 -> 169 us per call, half of
// it here).  Larger ones are the copy engine's, straight from and to the caller's buffer; ordinary
// memory is then staged by the driver (18 to 24 GB/s measured, which staging by several threads of our
// own did not beat at 0.6 to 2.2 MB: their wake-up costs more than they save).
#pragma once
#include "program.h"

namespace fluidml {
namespace worker {

class Transfer {
public:
  explicit Transfer(const Program &program) : program_(program) {}
  ~Transfer();
  // in[i] / out[i] belong to program.inputs[i] / program.outputs[i].
  void Begin(const std::vector<void *> &in, const std::vector<void *> &out);
  // Enqueues the copies of the inputs; page-locked buffers are read until the stream is done.
  void Upload(void *stream);
  // Enqueues what brings the outputs to the host ...
  void Download(void *stream);
  // ... and delivers them; the stream is synchronised when this returns.
  void Finish(void *stream);

private:
  struct Way { void *host; char *device; size_t offset, bytes, stage; bool small; };  // of one tensor; stage: place in the image
  struct Run { size_t offset, bytes, stage; };                                        // of small tensors side by side
  void Plan(const std::vector<IoBinding> &bindings, const std::vector<void *> &host, std::vector<Way> *ways, std::vector<Run> *runs,
            size_t *stage);
  const Program &program_;
  char *staging_ = nullptr;  // page-locked image of the runs
  size_t staging_bytes_ = 0;
  std::vector<Way> in_, out_;
  std::vector<Run> in_runs_, out_runs_;
};

}  // namespace worker
}  // namespace fluidml
