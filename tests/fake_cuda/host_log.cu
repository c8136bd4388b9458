// host_log.cu -- runs calls of the library's C ABI on the recording runtime (fake_cuda.cpp) and prints what
// they enqueue, for tests/test_host_launches.py. Compiled with the pass bodies left empty.
//
// TEST INFRASTRUCTURE ONLY. Usage: host_log create | reset | timeouts | settings | power W H split
#include "owl_api.cu"

#include <cstdlib>

extern "C" unsigned fake_next_word;
extern "C" std::string* fake_describe(const char* name, unsigned gridY, void** args) {
  const std::string n = name;
  auto* r = new std::string;
  if (n.find("k_pass") != 0) { return r; }
  *r = " timeout=";
  if (n.find("_group") != std::string::npos) {
    const auto* ga = static_cast<const owl::GroupArgs*>(args[0]);
    for (unsigned i = 0; i < gridY; ++i) { *r += (i ? "," : "") + std::to_string(ga->a[i].timeoutNs); }
  } else {
    *r += std::to_string(static_cast<const owl::Args*>(args[0])->timeoutNs);
  }
  return r;
}

namespace {
void must(int status) {
  if (status != OWL_OK) {
    std::printf("error %d %s\n", status, owl_last_error());
    std::exit(4);
  }
}
void mark(const char* s) { std::printf("== %s\n", s); }
owl_plan* plan(uint32_t W, uint32_t H, uint32_t split = 0) {
  owl_plan* p = nullptr;
  must(owl_plan_create(0, (uint32_t)(2.0 * W * H * 16.3) | 1, W, H, &p));
  must(owl_plan_set_split(p, (int)split));
  return p;
}
int32_t* buf(owl_plan* p) {
  int32_t* b = nullptr;
  must(owl_buf_alloc(p, &b));
  return b;
}
}  // namespace

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "create") {
    mark("create");
    owl_plan* p = nullptr;
    must(owl_plan_create(0, 133947, 64, 64, &p));
    mark("end");
  } else if (what == "reset") {
    owl_plan* p = plan(64, 64);
    mark("sync");
    fake_next_word = owl::DEVERR_WAIT;
    std::printf("status %d\n", owl_sync(p));
    mark("end");
  } else if (what == "timeouts") {
    owl_plan *p = plan(64, 64), *q = plan(64, 64), *r = plan(64, 128);
    int32_t *a = buf(p), *b = buf(p);
    int32_t* bufs[3] = {a, buf(q), buf(r)};
    owl_plan* plans[3] = {p, q, r};
    owl_batch* batch = nullptr;
    must(owl_batch_create(0, 3, plans, &batch));
    // limits that change, and come back, between calls that run as graphs
    for (uint64_t t : {7ull, 9ull, 7ull}) {
      must(owl_plan_set_timeout(p, t));
      must(owl_plan_set_timeout(r, t + 1));
      std::printf("== limit %llu\n", (unsigned long long)t);
      must(owl_square(p, b, a, 16, 0));
      float ms[3];
      uint32_t launches[3];
      must(owl_profile_square(p, a, 16, 0, ms, launches));
      for (int i = 0; i < 2; ++i) { must(owl_modmul(p, a, b, 0)); }
      mark("batch");
      must(owl_batch_square(batch, bufs, 3, 0));
    }
    mark("end");
  } else if (what == "settings") {
    owl_plan* p = plan(64, 2048);
    int32_t* a = buf(p);
    owl_batch* batch = nullptr;
    must(owl_batch_create(0, 1, &p, &batch));
    mark("plain");
    must(owl_batch_square(batch, &a, 3, 0));
    must(owl_plan_set_split(p, OWL_SPLIT_COLUMNS));
    mark("split");
    must(owl_batch_square(batch, &a, 3, 0));
    must(owl_plan_set_split(p, 0));
    must(owl_plan_set_column_variant(p, OWL_COL_V8));
    mark("variant");
    must(owl_batch_square(batch, &a, 3, 0));
    mark("end");
  } else if (what == "power" && argc == 5) {
    owl_plan* p = plan((uint32_t)std::atoi(argv[2]), (uint32_t)std::atoi(argv[3]), (uint32_t)std::atoi(argv[4]));
    int32_t *a = buf(p), *b = buf(p);
    mark("square");
    must(owl_square(p, b, a, 3, 0));
    mark("square without round-off");
    must(owl_square(p, b, a, 3, OWL_SQ_NO_ROE));
    mark("power");
    must(owl_exp_mul(p, a, 0xb5, b));
    for (int i = 0; i < 2; ++i) {
      mark("product");
      must(owl_modmul(p, a, b, 0));
    }
    mark("end");
  } else {
    return 2;
  }
  return 0;
}
