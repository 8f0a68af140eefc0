// Host code of the library on a CUDA runtime without a device (fake_cudart.cpp): error paths,
// launch shapes and choices by timing that no run on a GPU can bring about on purpose.
// usage: host_paths CASE (none: lists them); prints OK or the expectation that failed.
#include <sys/mman.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "fake_cudart.h"
#include "gems_b200.h"

namespace {

#define EXPECT(cond)                                            \
  do {                                                          \
    if (!(cond)) {                                              \
      std::printf("line %d: expected %s\n", __LINE__, #cond);   \
      std::exit(1);                                             \
    }                                                           \
  } while (0)

gems_session *session(int nstates, int ncat, int nptn, int precision, int scaling,
                      int ntaxa = 8) {
  gems_session_desc d{ntaxa, nptn, nstates, ncat, ntaxa, precision, scaling, 0};
  gems_session *s = nullptr;
  EXPECT(gems_session_create(&d, &s) == GEMS_OK);
  std::vector<uint8_t> tips((size_t)ntaxa * nptn, 1);
  EXPECT(gems_upload_tips(s, tips.data()) == GEMS_OK);
  std::vector<double> freq(nptn, 1.0), eval(nstates, -1.0), ev((size_t)nstates * nstates, 0.5);
  EXPECT(gems_upload_patterns(s, freq.data(), nullptr) == GEMS_OK);
  std::vector<double> r(ncat, 1.0), p(ncat, 1.0 / ncat);
  EXPECT(gems_set_model(s, eval.data(), ev.data(), ev.data(), r.data(), p.data()) == GEMS_OK);
  return s;
}

// slot k from tips: `n` updates
std::vector<gems_op> updates(int n) {
  std::vector<gems_op> ops;
  for (int k = 0; k < n; k++)
    ops.push_back(k == 0 ? gems_op{0, GEMS_CHILD_TIP, 0, GEMS_CHILD_TIP, 1, 0, 0.1, 0.1}
                         : gems_op{k, GEMS_CHILD_PARTIAL, k - 1, GEMS_CHILD_TIP, k + 1, 0, 0.1, 0.1});
  return ops;
}
const gems_branch kBranch{2, GEMS_CHILD_TIP, 5, 0, 0.1}, kOther{1, GEMS_CHILD_TIP, 6, 0, 0.1};

int count(const char *kernel) {
  int n = 0;
  for (const fake::Launch &l : fake::launches) n += l.kernel.find(kernel) != std::string::npos;
  return n;
}

std::map<std::string, void (*)()> &cases() {
  static std::map<std::string, void (*)()> m;
  return m;
}
#define CASE(name)                                                   \
  void name();                                                       \
  const bool name##_listed = (cases()[#name] = &name, true);         \
  void name()

// ---- an error that a call returned is not returned again by the next one --------------------
CASE(error_once) {
  gems_session *s = session(20, 4, 300, GEMS_PREC_FP64, GEMS_SCALE_SAFE);
  const std::vector<gems_op> ops = updates(3);
  double a, b;
  fake::fail_kernel = "k_terms";
  EXPECT(gems_branch_derv(s, ops.data(), 3, &kBranch, 1, &a, &b, nullptr) == GEMS_ERR_CUDA);
  fake::fail_kernel = "";
  EXPECT(gems_branch_derv(s, ops.data(), 3, &kBranch, 1, &a, &b, nullptr) == GEMS_OK);
  EXPECT(gems_session_destroy(s) == GEMS_OK);
}

// ---- a launch that forms theta and fails leaves no theta that a later call would read --------
void theta_after_failure(int nstates, int ncat, int precision, const char *kernel) {
  gems_session *s = session(nstates, ncat, 300, precision, GEMS_SCALE_SAFE);
  const std::vector<gems_op> ops = updates(3);
  double a, b;
  int n;
  for (int newton = 0; newton < 2; newton++) {
    auto form = [&](const gems_branch &br) {
      return newton ? gems_newton_branch(s, ops.data(), 3, &br, 1, 1e-6, 10.0, 1e-6, 5, &a, &n)
                    : gems_branch_derv(s, ops.data(), 3, &br, 1, &a, &b, nullptr);
    };
    EXPECT(form(kBranch) == GEMS_OK);
    EXPECT(gems_lnl_from_buffer(s, 0.1, &a, nullptr) == GEMS_OK);
    fake::fail_kernel = kernel[0] ? kernel : newton ? "k_newton" : "k_terms";
    EXPECT(form(kOther) == GEMS_ERR_CUDA);
    fake::fail_kernel = "";
    EXPECT(gems_lnl_from_buffer(s, 0.1, &a, nullptr) == GEMS_ERR_STATE);
    EXPECT(gems_branch_derv(s, nullptr, 0, &kBranch, 0, &a, &b, nullptr) == GEMS_ERR_STATE);
    EXPECT(gems_newton_branch(s, nullptr, 0, &kBranch, 0, 1e-6, 10.0, 1e-6, 5, &a, &n) ==
           GEMS_ERR_STATE);
    EXPECT(gems_get_theta(s, nullptr, nullptr) == GEMS_ERR_STATE);
    EXPECT(form(kOther) == GEMS_OK);
    EXPECT(gems_branch_derv(s, nullptr, 0, &kOther, 0, &a, &b, nullptr) == GEMS_OK);
  }
  EXPECT(gems_session_destroy(s) == GEMS_OK);
}
CASE(theta_4_fp64) { theta_after_failure(4, 4, GEMS_PREC_FP64, ""); }
CASE(theta_4_fp64_one_category) { theta_after_failure(4, 1, GEMS_PREC_FP64, ""); }
CASE(theta_4_mixed) { theta_after_failure(4, 4, GEMS_PREC_MIXED, ""); }
CASE(theta_20_fp64) { theta_after_failure(20, 4, GEMS_PREC_FP64, ""); }
CASE(theta_61_fp64) { theta_after_failure(61, 4, GEMS_PREC_FP64, ""); }
CASE(theta_20_mixed) { theta_after_failure(20, 4, GEMS_PREC_MIXED, "k_theta_mixed"); }

// ---- an ingest's results: a copy that fails leaves the caller's array as it was, and an address
// that the host cannot write to is an error of the copy -------------------------------------------
gems_ingest *ingest(int ntaxa, long long npat) {
  fake::on_launch = [npat](const std::string &name, void **args) {
    if (name.find("k_scan_sums") != std::string::npos) **static_cast<long long **>(args[2]) = npat;
  };
  std::vector<uint8_t> codes((size_t)ntaxa * npat);
  gems_ingest *g = nullptr;
  long long n = 0;
  EXPECT(gems_ingest_create(0, ntaxa, npat, 4, codes.data(), 1, &g, &n) == GEMS_OK && n == npat);
  return g;
}
CASE(ingest_failed_copy) {
  gems_ingest *g = ingest(64, 200000);
  std::vector<uint8_t> out((size_t)64 * 200000, 0xAB);
  fake::fail_call = "cudaMemcpy";
  EXPECT(gems_ingest_read(g, out.data(), nullptr, nullptr, nullptr) == GEMS_ERR_CUDA);
  fake::fail_call = "";
  for (uint8_t b : out) EXPECT(b == 0xAB);
  EXPECT(gems_ingest_read(g, out.data(), nullptr, nullptr, nullptr) == GEMS_OK);
  for (uint8_t b : out) EXPECT(b == 0);
  gems_ingest_destroy(g);
}
CASE(ingest_device_address) {
  gems_ingest *g = ingest(64, 200000);
  void *p = mmap(nullptr, (size_t)64 * 200000, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  EXPECT(p != MAP_FAILED);
  fake::device_only.insert(p);
  EXPECT(gems_ingest_read(g, static_cast<uint8_t *>(p), nullptr, nullptr, nullptr) ==
         GEMS_ERR_CUDA);
  gems_ingest_destroy(g);
}

// ---- kernel timing: every traversal counts under id 0, every theta under id 2 ------------------
void profile_counts(int nstates, int ncat, int precision) {
  gems_session *s = session(nstates, ncat, 300, precision, GEMS_SCALE_SAFE);
  const std::vector<gems_op> ops = updates(3);
  double a, b;
  int n;
  auto launches = [&](int id) {
    double ms = 0.0;
    long long k = 0;
    EXPECT(gems_profile_read(s, id, &ms, &k) == GEMS_OK);
    return (int)k;
  };
  EXPECT(gems_profile_enable(s, 1) == GEMS_OK);
  EXPECT(gems_branch_derv(s, ops.data(), 3, &kBranch, 1, &a, &b, nullptr) == GEMS_OK);
  EXPECT(launches(0) == 1 && launches(1) == 0 && launches(2) == 1 && launches(3) == 1);
  EXPECT(gems_newton_branch(s, ops.data(), 3, &kBranch, 1, 1e-6, 10.0, 1e-6, 5, &a, &n) ==
         GEMS_OK);
  EXPECT(launches(0) == 1 && launches(2) == 1 && launches(5) == 1);
  EXPECT(gems_lnl_from_buffer(s, 0.1, &a, nullptr) == GEMS_OK && launches(4) == 1);
  EXPECT(gems_branch_lnl(s, ops.data(), 3, &kBranch, &a, nullptr) == GEMS_OK);
  EXPECT(launches(0) == 1 && launches(1) == 1 && launches(2) == 0);
  EXPECT(gems_profile_enable(s, 0) == GEMS_OK);
  EXPECT(gems_branch_derv(s, ops.data(), 3, &kBranch, 1, &a, &b, nullptr) == GEMS_OK);
  for (int id = 0; id < 6; id++) EXPECT(launches(id) == 0);
  EXPECT(gems_session_destroy(s) == GEMS_OK);
}
CASE(profile_4_fp64) { profile_counts(4, 4, GEMS_PREC_FP64); }
CASE(profile_4_mixed) { profile_counts(4, 4, GEMS_PREC_MIXED); }
CASE(profile_20_fp64) { profile_counts(20, 4, GEMS_PREC_FP64); }
CASE(profile_20_mixed) { profile_counts(20, 4, GEMS_PREC_MIXED); }
CASE(profile_61_fp64) { profile_counts(61, 4, GEMS_PREC_FP64); }

// ---- Newton loops under a share of the GPU: within it, on as many SMs as its blocks can take ---
CASE(newton_share) {
  const std::vector<gems_op> ops = updates(3);
  double a;
  int n;
  for (int share : {2, 4, 16, 64})
    for (int form = 0; form < 3; form++) {
      const int states[] = {4, 20, 61}, cats[] = {8, 4, 16}, ptn[] = {400000, 100000, 20000};
      gems_session *s = session(states[form], cats[form], ptn[form], GEMS_PREC_FP64, GEMS_SCALE_SAFE);
      EXPECT(gems_session_set_option(s, GEMS_OPT_NEWTON_SHARE, share) == GEMS_OK);
      fake::launches.clear();
      EXPECT(gems_newton_branch(s, ops.data(), 3, &kBranch, 1, 1e-6, 10.0, 1e-6, 5, &a, &n) ==
             GEMS_OK);
      const fake::Launch &l = fake::launches.back();
      EXPECT(l.kernel.find("k_newton") != std::string::npos);
      const int blocks = (form == 0 ? 4 : 3) * 148 / share;  // of the blocks that fit the GPU
      EXPECT(l.grid <= blocks && l.grid >= std::min(256, blocks) / 8 * 8);
      EXPECT(gems_session_destroy(s) == GEMS_OK);
    }
}

// ---- FP64 20-state traversals of few patterns: four categories to a warp, not all of them -------
CASE(protein_few_patterns) {
  const std::vector<gems_op> ops = updates(3);
  for (int ncat = 1; ncat <= 16; ncat++)
    for (int ptn : {1, 100, 3000}) {
      gems_session *s = session(20, ncat, ptn, GEMS_PREC_FP64, GEMS_SCALE_NORM);
      fake::launches.clear();
      EXPECT(gems_traverse(s, ops.data(), 3) == GEMS_OK);
      const fake::Launch &l = fake::launches.back();
      EXPECT(l.kernel.find("k_traverse_f20") != std::string::npos);
      EXPECT(l.grid * l.threads / 32 >= (ptn + 7) / 8 * ((ncat + 3) / 4));
      EXPECT(gems_session_destroy(s) == GEMS_OK);
    }
}

// ---- the probe of the Newton loop's waits reports a time-out only when both ran out ------------
CASE(wait_probe) {
  for (int slots : {GEMS_OK, GEMS_ERR_TIMEOUT})
    for (int cluster : {GEMS_OK, GEMS_ERR_TIMEOUT}) {
      fake::on_launch = [=](const std::string &name, void **args) {
        if (name.find("k_exchange_probe") != std::string::npos) **static_cast<int **>(args[1]) = slots;
        if (name.find("k_cluster_probe") != std::string::npos) **static_cast<int **>(args[0]) = cluster;
      };
      int status = -1;
      EXPECT(gems_check_barrier_timeout(0, &status) == GEMS_OK);
      EXPECT((status == GEMS_ERR_TIMEOUT) == (slots && cluster));
    }
}

// ---- the launch shape of large 4-state traversals is chosen by the kernels' time: neither what the
// host does when a kernel is first used nor one launch that something else held up moves it ------
const char *tuned_kernel(int precision, double pattern_ms, double staged_ms, double first_use,
                         int held_up) {
  gems_session *s = session(4, 4, 200000, precision, GEMS_SCALE_NORM, 32);
  fake::first_use_ms = [=](const std::string &name) {  // the first of them loads the most
    return name.find("k_traverse4p") != std::string::npos ? first_use : 0.5;
  };
  int full = 0;
  fake::kernel_ms = [&](const std::string &name, const fake::Launch &l) {
    const bool pattern = name.find("k_traverse4p") != std::string::npos;
    if (!pattern && name.find("k_traverse4q") == std::string::npos) return 0.01;
    if (l.grid < 100) return 0.5;  // a few patterns
    if (pattern && full++ < held_up) return 30.0;
    return pattern ? pattern_ms : staged_ms;
  };
  const std::vector<gems_op> ops = updates(31);
  EXPECT(gems_traverse(s, ops.data(), 31) == GEMS_OK);
  fake::launches.clear();
  EXPECT(gems_traverse(s, ops.data(), 31) == GEMS_OK);
  EXPECT(count("k_traverse4p") + count("k_traverse4q") == 1);  // tuned: one launch
  const char *k = count("k_traverse4p") ? "pattern" : "staged";
  EXPECT(gems_session_destroy(s) == GEMS_OK);
  return k;
}
CASE(tuner_first_use) {
  EXPECT(!std::strcmp(tuned_kernel(GEMS_PREC_MIXED, 6.0, 13.0, 25.0, 0), "pattern"));
  EXPECT(!std::strcmp(tuned_kernel(GEMS_PREC_FP64, 6.0, 13.0, 25.0, 0), "pattern"));
}
CASE(tuner_held_up) {
  EXPECT(!std::strcmp(tuned_kernel(GEMS_PREC_MIXED, 6.0, 13.0, 0.0, 1), "pattern"));
}
CASE(tuner_faster_shape) {
  EXPECT(!std::strcmp(tuned_kernel(GEMS_PREC_MIXED, 13.0, 6.0, 25.0, 0), "staged"));
  EXPECT(!std::strcmp(tuned_kernel(GEMS_PREC_FP64, 6.0, 5.95, 25.0, 0), "pattern"));  // within noise
}

// a list that reads a slot and then writes it gives something else when it is run again: not tuned
CASE(tuner_list_not_repeatable) {
  gems_session *s = session(4, 4, 200000, GEMS_PREC_FP64, GEMS_SCALE_NORM, 32);
  auto launches = [&](const std::vector<gems_op> &ops) {
    fake::launches.clear();
    EXPECT(gems_traverse(s, ops.data(), (int)ops.size()) == GEMS_OK);
    return count("k_traverse4") + count("k_traverse_f64x");
  };
  std::vector<gems_op> ops = updates(31);
  ops[0].left_kind = GEMS_CHILD_PARTIAL, ops[0].left_id = 30;  // as it was: written by the last op
  EXPECT(launches(ops) == 1);
  ops[0].left_id = 31;  // not written
  EXPECT(launches(ops) > 1);
  EXPECT(launches(ops) == 1);
  EXPECT(gems_session_destroy(s) == GEMS_OK);
}

// ---- a session's footprint is what it allocates --------------------------------------------------
CASE(footprint) {
  for (int nstates : {4, 20, 61})
    for (int precision : {GEMS_PREC_FP64, GEMS_PREC_MIXED})
      for (int ncat : {1, 4, 16}) {
        gems_session_desc d{12, 777, nstates, ncat, 10, precision, GEMS_SCALE_SAFE, 0};
        size_t bytes = 0;
        EXPECT(gems_session_footprint(&d, &bytes) == GEMS_OK);
        gems_session *s = nullptr;
        EXPECT(gems_session_create(&d, &s) == GEMS_OK);
        EXPECT(bytes == fake::allocated);
        EXPECT(gems_session_destroy(s) == GEMS_OK);
        EXPECT(fake::allocated == 0);
      }
}

// ---- a module is loaded whole by the first launch of one of its kernels: the branch kernels, most
// of the library's, come in modules of one kind of session each -----------------------------------
CASE(branch_modules) {
  int branch = 0;
  for (const auto &m : fake::modules()) {
    int here = 0;
    for (const std::string &k : m.second)
      here += k.find("k_terms") != std::string::npos || k.find("k_newton") != std::string::npos;
    EXPECT(here <= 12);
    branch += here;
  }
  EXPECT(branch >= 50);
}

}  // namespace

int main(int argc, char **argv) {
  if (argc == 1) {
    for (const auto &c : cases()) std::printf("%s\n", c.first.c_str());
    return 0;
  }
  const auto it = cases().find(argv[1]);
  if (it == cases().end()) return 2;
  it->second();
  std::printf("OK\n");
  return 0;
}
