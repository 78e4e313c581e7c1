// batch_host_check.cu — test driver for the host side of batch.cu (items, budget,
// errors), linked with that file, fake_cudart.cpp in place of the CUDA runtime and
// the fakes below in place of the library's other sources.  Usage:
// batch_host_check <command> <budget> <fail_at> <sector>... with sectors as
// fft:phased:frames:count.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>
#include <vector>

#include "fake_cudart.h"
#include "fxc.h"
#include "fxc_internal.h"
#include "fxc_kernels.h"

using namespace fxc;

struct fxc_engine {
  uint64_t budget = ~0ull, in_use = 0;
} g_engine;
struct fxc_scan {
  uint32_t n;
  bool phased;
};

namespace {

struct Launch {
  std::string name;
  int group;
  cudaStream_t stream;
  std::set<int> before;
  std::vector<BatchItem> items;
  std::vector<uint32_t> flush;  // per item: its sector's flush interval
};
std::vector<Launch> g_log;
int g_fail_at = -1;
std::string g_msg;

cudaError_t launch(const char* name, int group, const BatchArgs& a, cudaStream_t s) {
  const int id = (int)g_log.size();
  Launch l{name, group, s, of(s).before, {}, {}};
  if (group >= 0) {
    for (uint32_t k = 0; k < a.hdr->nitems[group]; ++k) {
      const BatchItem& it = a.hdr->items[a.hdr->item0[group] + k];
      const BatchScan& b = a.hdr->scans[it.scan];
      l.items.push_back(it);
      l.flush.push_back(b.phased ? b.pp.flush_every : b.p.flush_every);
    }
  }
  g_log.push_back(l);
  if (id == g_fail_at) {
    g_log[id].name += "!";
    return cudaErrorLaunchFailure;
  }
  of(s).before.insert(id);
  return cudaSuccess;
}

}  // namespace

// ---- the library's other sources
namespace fxc {
fxc_status internal_fail(fxc_status s, const char* msg) {
  g_msg = msg;
  return s;
}
int engine_sm_count(const fxc_engine*) { return 148; }
int engine_device(const fxc_engine*) { return 0; }
fxc_engine* scan_engine(const fxc_scan*) { return &g_engine; }
fxc_status engine_reserve(fxc_engine* e, uint64_t bytes) {
  if (e->in_use + bytes > e->budget) return internal_fail(FXC_EBUSY, "HBM budget exhausted");
  e->in_use += bytes;
  return FXC_OK;
}
void engine_release(fxc_engine* e, uint64_t bytes) { e->in_use -= bytes; }
void engine_track_batch(fxc_engine*, fxc_batch*, bool) {}
fxc_status batch_describe(fxc_scan* s, const uint8_t*, const uint8_t*, uint64_t nf, uint64_t,
                          double*, uint8_t*, BatchScan* out, int* group) {
  static const uint32_t len[] = {1024, 2048, 4096, 8192, 16384};
  BatchScan b{};
  b.p.nf = b.pp.nf = nf;
  b.p.flush_every = b.pp.flush_every = s->n < 4096 ? s->n / 128 : 32;  // 32 frames of its own kernel
  b.n = s->n;
  b.h = s->n / 2 + 1;
  b.phased = s->phased ? 1 : 0;
  *out = b;
  for (int k = 0; k < 5; ++k)
    if (len[k] == s->n) *group = k + (s->phased ? kCorrGroups : 0);
  return FXC_OK;
}
fxc_status run_sector_internal(fxc_scan*, const uint8_t*, const uint8_t*, uint64_t, uint64_t,
                               double*, uint8_t*, cudaStream_t) {
  return FXC_EINVAL;  // no sector here takes the per-scan path
}
cudaError_t batch_prepare(int, int) { return cudaSuccess; }
int batch_group_ctas_per_sm(int g, int) { return g < BG_8192 ? 2 : 1; }
cudaError_t launch_batch_group(int g, int, const BatchArgs& a, int, cudaStream_t s) {
  return launch("corr", g, a, s);
}
cudaError_t launch_batch_frame_info(const BatchArgs& a, int, cudaStream_t s) {
  return launch("records", -1, a, s);
}
cudaError_t launch_batch_reduce(const BatchArgs& a, int, cudaStream_t s) {
  return launch("reduce", -1, a, s);
}
cudaError_t phased_batch_prepare(uint32_t) { return cudaSuccess; }
int phased_batch_ctas_per_sm(uint32_t n) { return n < 8192 ? 2 : 1; }
int phased_frames_per_cta_iter(uint32_t n) { return n == 1024 ? 4 : (n == 2048 ? 2 : 1); }
cudaError_t launch_phased_batch(uint32_t, const BatchArgs& a, int g, int, cudaStream_t s) {
  return launch("phased", g, a, s);
}
}  // namespace fxc
extern "C" {
const char* fxc_last_error() { return g_msg.c_str(); }
uint64_t fxc_bytes_per_frame(uint32_t n, uint32_t bits) { return (uint64_t)n * bits / 8; }
fxc_status fxc_scan_open(fxc_engine*, const fxc_scan_cfg* c, fxc_scan** out) {
  *out = new fxc_scan{c->fft_len, false};
  return FXC_OK;
}
fxc_status fxc_scan_close(fxc_scan* s) {
  delete s;
  return FXC_OK;
}
}

namespace {

struct Call {
  std::vector<fxc_scan*> scans;
  std::vector<const uint8_t*> raw;
  std::vector<uint64_t> nf, first;
  std::vector<double*> acc;
  std::vector<uint8_t*> out;
};

fxc_status run(fxc_batch* b, Call& c, cudaStream_t s) {
  return fxc_batch_run_device_raw(b, c.scans.data(), c.raw.data(), c.raw.data(), c.nf.data(),
                                  c.first.data(), c.acc.data(), c.out.data(),
                                  (uint32_t)c.scans.size(), s);
}

// One line a launch: name, group, the launches before it; with `items`, those too.
void print_log(bool items) {
  for (size_t k = 0; k < g_log.size(); ++k) {
    const Launch& l = g_log[k];
    std::printf("%zu %s %d before", k, l.name.c_str(), l.group);
    for (int x : l.before) std::printf(" %d", x);
    if (items)
      for (size_t i = 0; i < l.items.size(); ++i)
        std::printf("\n  item %u %u %llu %llu %llu %u %u", l.items[i].scan, l.items[i].row,
                    (unsigned long long)l.items[i].f0, (unsigned long long)l.items[i].f1,
                    (unsigned long long)l.items[i].part, l.items[i].slots, l.flush[i]);
    std::printf("\n");
  }
}

}  // namespace

int main(int argc, char** argv) {
  const std::string cmd = argv[1];
  const uint64_t budget = std::strtoull(argv[2], nullptr, 10);
  g_fail_at = std::atoi(argv[3]);
  Call c;
  for (int k = 4; k < argc; ++k) {
    unsigned n, ph, nf, count;
    if (std::sscanf(argv[k], "%u:%u:%u:%u", &n, &ph, &nf, &count) != 4) return 2;
    for (unsigned i = 0; i < count; ++i) {
      c.scans.push_back(new fxc_scan{n, ph != 0});
      c.nf.push_back(nf);
    }
  }
  const size_t m = c.scans.size();
  c.raw.resize(m);
  c.first.resize(m);
  c.acc.resize(m);
  c.out.resize(m);
  fxc_batch* b = nullptr;
  if (fxc_batch_create(&g_engine, nullptr, &b) != FXC_OK) return 3;
  cudaStream_t s[2];
  for (auto& x : s) cudaStreamCreateWithFlags(&x, 0);
  if (budget) g_engine.budget = budget;
  if (cmd == "shape" || cmd == "pinned")  // a shape of the caller's
    if (fxc_batch_set_shape(b, c.scans[0]->n, 1, 64) != FXC_OK) return 3;
  if (cmd == "pinned") {  // then the tuner's
    if (fxc_batch_autotune(b, c.scans[0]->n) != FXC_OK) return 3;
    g_log.clear();
  }
  const fxc_status st = run(b, c, s[0]);
  std::printf("status %d\n", (int)st);
  if (cmd == "error") {
    // what the caller's stream and the next call, on another stream, wait for
    std::printf("stream");
    for (int x : of(s[0]).before) std::printf(" %d", x);
    g_fail_at = -1;
    std::printf("\nagain %d\n", (int)run(b, c, s[1]));
  }
  std::printf("in_use %llu\n", (unsigned long long)g_engine.in_use);
  print_log(cmd != "error");
  fxc_batch_destroy(b);
  std::printf("left %llu\n", (unsigned long long)g_engine.in_use);
  return 0;
}
