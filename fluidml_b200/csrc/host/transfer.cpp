#include "transfer.h"
#include <algorithm>
#include <cstring>

namespace fluidml {
namespace worker {

namespace {
constexpr size_t kSmall = 64 * 1024;

void Check(int status, const char *what) {
  if (status != FML_OK) throw Error(std::string(what) + ": " + fml_last_error());
}
}  // namespace

Transfer::~Transfer() {
  if (staging_) fml_host_free_pinned(staging_);
}

void Transfer::Plan(const std::vector<IoBinding> &bindings, const std::vector<void *> &host, std::vector<Way> *ways,
                    std::vector<Run> *runs, size_t *stage) {
  ways->clear();
  runs->clear();
  for (size_t i = 0; i < host.size(); ++i) {
    const IoBinding &b = bindings[i];
    Way w;
    w.host = host[i];
    w.device = static_cast<char *>(b.device);
    w.offset = (size_t)(w.device - static_cast<const char *>(program_.io));
    w.bytes = b.bytes;
    w.small = b.bytes <= kSmall;
    w.stage = 0;
    if (w.small) {
      // tensors start on 256-byte steps of the interface block: neighbours are at most that far apart
      Run *r = runs->empty() ? nullptr : &runs->back();
      if (r && w.offset >= r->offset + r->bytes && w.offset - (r->offset + r->bytes) < 256 && w.offset + w.bytes - r->offset <= 4 * kSmall) {
        r->bytes = w.offset + w.bytes - r->offset;
      } else {
        runs->push_back({w.offset, w.bytes, *stage});
        r = &runs->back();
      }
      w.stage = r->stage + (w.offset - r->offset);
      *stage = (w.stage + w.bytes + 255) / 256 * 256;
    }
    ways->push_back(w);
  }
}

void Transfer::Begin(const std::vector<void *> &in, const std::vector<void *> &out) {
  size_t need = 0;
  Plan(program_.inputs, in, &in_, &in_runs_, &need);
  Plan(program_.outputs, out, &out_, &out_runs_, &need);
  if (need <= staging_bytes_) return;
  // (no copy of this object is in flight: every run ends synchronised)
  if (staging_) Check(fml_host_free_pinned(staging_), "freeing the staging memory");
  staging_ = nullptr;
  staging_bytes_ = 0;
  void *p = nullptr;
  Check(fml_host_alloc_pinned(&p, need), "allocating the staging memory");
  staging_ = static_cast<char *>(p);
  staging_bytes_ = need;
}

void Transfer::Upload(void *stream) {
  for (const Way &w : in_) {
    if (w.small) memcpy(staging_ + w.stage, w.host, w.bytes);
    else Check(fml_memcpy_h2d(w.device, w.host, w.bytes, stream), "copying an input");
  }
  for (const Run &r : in_runs_)
    Check(fml_copy_small((char *)program_.io + r.offset, staging_ + r.stage, r.bytes, stream), "copying the inputs");
}

void Transfer::Download(void *stream) {
  for (const Run &r : out_runs_)
    Check(fml_copy_small(staging_ + r.stage, (char *)program_.io + r.offset, r.bytes, stream), "copying the outputs");
  for (const Way &w : out_)
    if (!w.small) Check(fml_memcpy_d2h(w.host, w.device, w.bytes, stream), "copying an output");
}

void Transfer::Finish(void *stream) {
  Check(fml_stream_sync(stream), "waiting for the pass");
  for (const Way &w : out_)
    if (w.small) memcpy(w.host, staging_ + w.stage, w.bytes);
}

}  // namespace worker
}  // namespace fluidml
