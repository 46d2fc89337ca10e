// Runtime and C ABI for single transforms.
//
// Replaces the host launcher best_fft (cuda/fft_kernel.cu:117-147): that one
// prints, asserts n == 2^16, ignores omg, cudaMallocs two buffers per call
// that it never frees, launches one fixed <<<5,256>>> grid and exits the
// process on a launch error.  Here a call validates its arguments, resolves
// device-resident twiddle tables (built once per (field, root) and cached),
// enqueues one kernel per pass on the caller's stream and returns an error
// code on any failure.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <string>
#include <tuple>
#include <vector>

#include "gpusnarks_gb300.h"
#include "runtime.h"

namespace gsn {

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------
static thread_local std::string t_error;

int set_error(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  t_error = buf;
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  cudaGetLastError();  // a failed call leaves its error there, and the next launch would report it as its own
  return set_error(GSN_ERR_CUDA, "%s failed: %s (%d)", what, cudaGetErrorString(e), (int)e);
}

static std::atomic<uint64_t> g_launches{0};
void count_launches(uint64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return dev;
}

// SM count of the current device, looked up once per device.
int current_device_sms() {
  constexpr int kDevices = 64;
  static std::atomic<int> sms[kDevices];
  const int dev = current_device();
  if (dev < 0 || dev >= kDevices) return 1;
  int v = sms[dev].load(std::memory_order_relaxed);
  if (v <= 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) {
      cudaGetLastError();
      v = 1;
    }
    sms[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

const FieldOps* field_ops(int field) {
  switch (field) {
    case GSN_P32: return &kOpsP32;
    case GSN_BLS12_381_FR: return &kOpsBLS12_381;
    case GSN_MNT4753_FR: return &kOpsMNT4_753;
    default: return nullptr;
  }
}

// ---------------------------------------------------------------------------
// device allocations
// ---------------------------------------------------------------------------
// The thread's last failed allocation found no memory: cudaMalloc also fails while another thread captures, and freeing
// or remembering anything for that would be wrong.
static thread_local bool t_no_memory = false;

static int dev_alloc_plain(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes ? bytes : 16);
  t_no_memory = e == cudaErrorMemoryAllocation;
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return set_error(GSN_ERR_NOMEM, "cudaMalloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
  }
  return GSN_OK;
}

void dev_free(void* p) {
  if (p) cudaFree(p);
}

// ---------------------------------------------------------------------------
// plans
// ---------------------------------------------------------------------------
struct FieldLimits {
  int max_r, target_j, max_block;
};

static FieldLimits limits_of(const FieldOps& F) {
  switch (F.id) {
    case GSN_P32: return {11, 3, 512};
    case GSN_BLS12_381_FR: return {8, 2, 128};
    default: return {8, 1, 128};
  }
}

size_t plan_smem_bytes(const FieldOps& F, const Plan& p, int pass) {
  return tile_words(F.limbs, (uint64_t)1 << (p.radix_log[pass] + p.log_j[pass])) * sizeof(uint32_t);
}

bool plan_valid(const FieldOps& F, const Plan& p) {
  if (p.npass < 1 || p.npass > kMaxPasses) return false;
  if (p.kernel == kKernelP32) {
    // 16-byte vectors along 4..16 columns, at least two passes, radix >= 4
    if (F.id != GSN_P32 || p.npass < 2 || (p.e_log != 3 && p.e_log != 4)) return false;
    for (int i = 0; i < p.npass; ++i)
      if (p.log_j[i] < 2 || p.log_j[i] > 4 || p.radix_log[i] < 2 || p.block[i] > 512) return false;
  } else if (p.kernel == kKernelRB) {
    // at most 4 columns per tile, sub-steps of 4 or 8 rows: what tables that name this kernel hold
    if (F.id != GSN_BLS12_381_FR || (p.e_log != 2 && p.e_log != 3)) return false;
    for (int i = 0; i < p.npass; ++i)
      if (p.log_j[i] > 2 || p.radix_log[i] < 1 || p.block[i] > 256) return false;
  } else if (p.kernel == kKernelLanes) {
    if (F.id != GSN_MNT4753_FR) return false;
  } else if (p.kernel != kKernelGeneric) {
    return false;
  }
  int sum = 0;
  for (int i = 0; i < p.npass; ++i) {
    if (p.radix_log[i] < 0 || p.log_j[i] < 0) return false;
    sum += p.radix_log[i];
    if (p.block[i] < 32 || p.block[i] > 1024 || (p.block[i] & 31)) return false;
    if (plan_smem_bytes(F, p, i) > 200 * 1024) return false;
  }
  if (sum != p.log_n) return false;
  for (int i = 0; i < p.npass; ++i) {
    const bool last = i == p.npass - 1;
    int inner = 0;
    for (int k = i + 1; k < p.npass; ++k) inner += p.radix_log[k];
    if (!last && p.log_j[i] > inner) return false;
    if (last && p.npass > 1 && p.log_j[i] > p.radix_log[0]) return false;
    if (last && p.npass == 1 && p.log_j[i] != 0) return false;
  }
  return true;
}

// Tile widths and threads per pass for a plan whose pass radices are set.
static void fill_tiles(Plan& p, int target_j, int max_block) {
  for (int i = 0; i < p.npass; ++i) {
    const bool last = i == p.npass - 1;
    int inner = 0;
    for (int k = i + 1; k < p.npass; ++k) inner += p.radix_log[k];
    int lj = last ? (p.npass == 1 ? 0 : std::min(target_j, p.radix_log[0])) : std::min(target_j, inner);
    p.log_j[i] = lj;
    int work = std::max(1, (1 << (p.radix_log[i] + lj)) / 2);
    int blk = 32;
    while (blk < max_block && blk < work) blk *= 2;
    p.block[i] = blk;
  }
}

Plan make_plan(const FieldOps& F, int log_n, int max_r, int target_j, int max_block) {
  Plan p;
  p.log_n = log_n;
  p.npass = std::max(1, (log_n + max_r - 1) / max_r);
  if (p.npass > kMaxPasses) p.npass = kMaxPasses;
  const int base = log_n / p.npass, extra = log_n % p.npass;
  for (int i = 0; i < p.npass; ++i) p.radix_log[i] = base + (i < extra ? 1 : 0);
  fill_tiles(p, target_j, max_block);
  (void)F;
  return p;
}

Plan make_split_plan(const FieldOps& F, int log_n, const int* radix_log, int npass, int target_j, int max_block) {
  Plan p;
  p.log_n = log_n;
  p.npass = std::min(npass, kMaxPasses);
  for (int i = 0; i < p.npass; ++i) p.radix_log[i] = radix_log[i];
  fill_tiles(p, target_j, max_block);
  (void)F;
  return p;
}

static void forget_calls();

static std::mutex g_plan_mu;
// (field, log_n, mode) -> plan; mode 0 = single transforms, 1 = batched kernel
static std::map<std::tuple<int, int, int>, Plan> g_tuned;

void set_tuned_plan(int field, int log_n, const Plan& p, int mode) {
  {
    std::lock_guard<std::mutex> g(g_plan_mu);
    g_tuned[std::make_tuple(field, log_n, mode)] = p;
  }
  forget_calls();
}
void clear_tuned_plans() {
  {
    std::lock_guard<std::mutex> g(g_plan_mu);
    g_tuned.clear();
  }
  forget_calls();
}
bool get_tuned_plan(int field, int log_n, Plan* out, int mode) {
  std::lock_guard<std::mutex> g(g_plan_mu);
  auto it = g_tuned.find(std::make_tuple(field, log_n, mode));
  if (it == g_tuned.end()) return false;
  *out = it->second;
  return true;
}

// Register-blocked 32-bit plan: passes of radix <= 2^max_r over tiles of
// 2^log_j columns, 2^e_log rows per thread per register sub-step.
Plan make_p32_plan(int log_n, int max_r, int log_j, int e_log) {
  Plan p;
  p.log_n = log_n;
  p.kernel = kKernelP32;
  p.e_log = e_log;
  p.npass = std::max(2, (log_n + max_r - 1) / max_r);
  if (p.npass > kMaxPasses) p.npass = kMaxPasses;
  const int base = log_n / p.npass, extra = log_n % p.npass;
  for (int i = 0; i < p.npass; ++i) p.radix_log[i] = base + (i < extra ? 1 : 0);
  for (int i = 0; i < p.npass; ++i) {
    const bool last = i == p.npass - 1;
    int inner = 0;
    for (int k = i + 1; k < p.npass; ++k) inner += p.radix_log[k];
    const int lj = std::min(log_j, last ? p.radix_log[0] : inner);
    p.log_j[i] = lj;
    int threads = (1 << (p.radix_log[i] + lj)) >> (2 + e_log);
    threads = std::max(32, std::min(512, threads));
    p.block[i] = threads;
  }
  return p;
}

Plan plan_for(const FieldOps& F, int log_n, bool batched) {
  Plan p;
  // batched plans come from their own table: a persistent launch runs every
  // tile with the batch's largest block, so it wants wider tiles than a
  // lone transform does
  const int mode = batched ? 1 : 0;
  if (get_tuned_plan(F.id, log_n, &p, mode) && plan_valid(F, p) && (!batched || p.kernel == kKernelGeneric))
    return p;
  if (F.id == GSN_P32 && !batched && log_n >= 8) {
    // tiles of at most 2^14 elements (64 KB): J = 8 columns, radix <= 2^11
    p = make_p32_plan(log_n, 11, 3, 4);
    if (plan_valid(F, p)) return p;
  }
  FieldLimits L = limits_of(F);
  return make_plan(F, log_n, L.max_r, L.target_j, L.max_block);
}

// ---------------------------------------------------------------------------
// twiddle / coset table cache
// ---------------------------------------------------------------------------
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
};

// A table in device memory, freed with its last holder.
struct Table {
  void* p = nullptr;
  size_t bytes = 0;
  uint64_t born = 0;  // four-step factors: TableCache::births when they were built
  ~Table() { dev_free(p); }
};
using TableRef = std::shared_ptr<const Table>;

struct PassTables {
  const uint32_t* stage[kMaxPasses] = {nullptr, nullptr, nullptr, nullptr};
  const uint32_t* step[kMaxPasses] = {nullptr, nullptr, nullptr, nullptr};
  uint64_t born = 0;
  bool stages_only = false;  // a caller's root, seen once: without its four-step factors
  bool none = false;  // there was no memory for them: the full table is read until tables are given back
  std::vector<std::shared_ptr<const void>> held;
};
struct Call;

// Every entry belongs to the device that was current when it was built: tables and scratch are keyed by
// device as well, so a process that drives several GPUs never hands one GPU another's memory.
struct TableCache {
  std::mutex mu;
  // (device, field, tw_log, root limbs) -> powers of the root
  struct Powers {
    TableRef table;
    bool pinned;  // default roots, and what gsn_prepare or a server's warm-up asked for
  };
  std::map<std::tuple<int, int, int, std::string>, Powers> powers;
  // (device, field, log2 of the order, r, name of the root) -> four-step factors of a pass of radix 2^r; r = kStage: the
  // stage twiddles of that order.  The name is empty for the default roots, else the caller's root and its order.
  std::map<std::tuple<int, int, int, int, std::string>, TableRef> steps;
  // (device, field, log_n, split, root limbs) -> the pass tables above, one lookup per call
  std::map<std::tuple<int, int, int, std::string>, std::shared_ptr<const PassTables>> passes;
  std::set<std::shared_ptr<const Call>> captured;  // what captured graphs run, kept until the caches are released
  std::map<std::tuple<int, cudaStream_t, int>, DevBuf> scratch;
  std::map<int, cudaStream_t> gen_stream;  // per device
  uint64_t births = 0;                     // pass tables and their factors built so far
  std::map<int, size_t> memory;            // per device: its memory in bytes
};

static TableCache& cache() {
  static TableCache* c = new TableCache();  // never destroyed: outlives static teardown order
  return *c;
}

static bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (s && cudaStreamIsCapturing(s, &cap) != cudaSuccess) cudaGetLastError();
  return cap != cudaStreamCaptureStatusNone;
}

// Frees the current device's tables that nobody holds, except pinned ones: the tables of roots and shifts that no call,
// batch or captured graph is using, and all pass tables out of use.  They are rebuilt when they are next needed.  Caller
// holds C.mu, so nobody takes a reference meanwhile; work already enqueued on them is waited for.  False: nothing freed.
static bool give_back_tables(TableCache& C) {
  const int dev = current_device();
  forget_calls();  // the look-up's own references
  std::atomic_thread_fence(std::memory_order_acquire);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  size_t freed = 0;
  for (auto it = C.passes.begin(); it != C.passes.end();)
    it = std::get<0>(it->first) == dev && (it->second->none || it->second.use_count() == 1) ? C.passes.erase(it)
                                                                                            : std::next(it);
  for (auto it = C.steps.begin(); it != C.steps.end();) {
    if (std::get<0>(it->first) == dev && it->second.use_count() == 1) {
      freed += it->second->bytes;
      it = C.steps.erase(it);
    } else {
      ++it;
    }
  }
  for (auto it = C.powers.begin(); it != C.powers.end();) {
    if (std::get<0>(it->first) == dev && !it->second.pinned && it->second.table.use_count() == 1) {
      freed += it->second.table->bytes;
      it = C.powers.erase(it);
    } else {
      ++it;
    }
  }
  return freed > 0;
}

// Room for a table of `need` bytes within half of the device's memory, which bounds what is kept of roots and shifts that
// may never come again (pinned tables do not count).  At the bound everything out of use goes at once: a drain per
// thousand tables of 2^20 elements, where dropping the oldest would drain for each.
static bool table_room(TableCache& C, size_t need, cudaStream_t s) {
  const int dev = current_device();
  size_t& total = C.memory[dev];
  if (total == 0) {
    size_t avail = 0;
    if (cudaMemGetInfo(&avail, &total) != cudaSuccess) {
      cudaGetLastError();
      total = 0;
      return true;
    }
  }
  auto fits = [&] {
    size_t kept = need;
    for (const auto& kv : C.steps)
      if (std::get<0>(kv.first) == dev) kept += kv.second->bytes;
    for (const auto& kv : C.powers)
      if (std::get<0>(kv.first) == dev && !kv.second.pinned) kept += kv.second.table->bytes;
    return kept <= total / 2;
  };
  if (fits()) return true;
  if (capturing(s)) return false;
  give_back_tables(C);
  return fits();
}

// dev_alloc with C.mu held, for a call on stream `s` (nothing is given back under capture).
static int dev_alloc_locked(TableCache& C, void** p, size_t bytes, cudaStream_t s) {
  int rc = dev_alloc_plain(p, bytes);
  if (rc == GSN_ERR_NOMEM && t_no_memory && !capturing(s) && give_back_tables(C)) rc = dev_alloc_plain(p, bytes);
  return rc;
}

int dev_alloc(void** p, size_t bytes) {
  int rc = dev_alloc_plain(p, bytes);
  if (rc != GSN_ERR_NOMEM || !t_no_memory) return rc;
  TableCache& C = cache();
  std::lock_guard<std::mutex> g(C.mu);
  return give_back_tables(C) ? dev_alloc_plain(p, bytes) : rc;
}

static std::string limbs_key(const uint32_t* x, int n) {
  return std::string(reinterpret_cast<const char*>(x), sizeof(uint32_t) * n);
}

// g^((p-1)/2^log_n), memoised: the exponentiation costs up to ~1 ms on the
// host for the 753-bit field and every call needs it.
static void default_root(const FieldOps& F, int log_n, uint32_t* out) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, std::string> memo;
  std::lock_guard<std::mutex> g(mu);
  auto key = std::make_pair(F.id, log_n);
  auto it = memo.find(key);
  if (it == memo.end()) {
    uint32_t r[kMaxLimbs];
    F.root(log_n, r);
    it = memo.emplace(key, limbs_key(r, F.limbs)).first;
  }
  std::memcpy(out, it->second.data(), it->second.size());
}

// Field inverse (canonical in and out), memoised: one costs a full host exponentiation (about a
// millisecond for the 753-bit field), and every coset-inverse transform needs s^-1.
static void inv_memo(const FieldOps& F, const uint32_t* x, uint32_t* out) {
  static std::mutex mu;
  static std::map<std::pair<int, std::string>, std::string> memo;
  const std::string key = limbs_key(x, F.limbs);
  std::lock_guard<std::mutex> g(mu);
  auto it = memo.find(std::make_pair(F.id, key));
  if (it == memo.end()) {
    uint32_t r[kMaxLimbs] = {0};
    F.inv(x, r);
    it = memo.emplace(std::make_pair(F.id, key), limbs_key(r, F.limbs)).first;
  }
  std::memcpy(out, it->second.data(), it->second.size());
}

// Returns a cached table of base^e for e in [0, 2^log_count), entries as
// fe_mul_tw takes them, held by T; builds it on first use.  Caller holds no lock.
static int powers_table(const FieldOps& F, const uint32_t* base, int log_count, const uint32_t** out, Tables* T,
                        cudaStream_t s, bool pin) {
  TableCache& C = cache();
  const int dev = current_device();
  std::lock_guard<std::mutex> g(C.mu);
  auto key = std::make_tuple(dev, F.id, log_count, limbs_key(base, F.limbs));
  auto it = C.powers.find(key);
  if (it == C.powers.end()) {
    cudaStream_t& gen = C.gen_stream[dev];
    if (!gen) GSN_CUDA(cudaStreamCreateWithFlags(&gen, cudaStreamNonBlocking));
    const uint64_t count = (uint64_t)1 << log_count;
    auto b = std::make_shared<Table>();
    b->bytes = table_words(F, count) * sizeof(uint32_t);
    if (!pin) table_room(C, b->bytes, s);  // held tables may be more than the bound
    int rc = dev_alloc_locked(C, &b->p, b->bytes, s);
    if (rc) return rc;
    cudaError_t e = F.powers(static_cast<uint32_t*>(b->p), count, base, gen);
    if (e == cudaSuccess) e = cudaStreamSynchronize(gen);
    if (e != cudaSuccess) return cuda_fail(e, "twiddle generation");
    count_launches(1);
    it = C.powers.emplace(key, TableCache::Powers{b, false}).first;
  }
  it->second.pinned = it->second.pinned || pin;
  T->held.push_back(it->second.table);
  *out = static_cast<const uint32_t*>(it->second.table->p);
  return GSN_OK;
}

// The default root table covering log_n: reuse any cached default table of
// order >= 2^log_n (its powers include every smaller root's), else build one
// of order 2^max(log_n, default_tw_log).
static int default_twiddles(const FieldOps& F, int log_n, const uint32_t** tw, int* tw_log, Tables* T, cudaStream_t s) {
  if (find_default_twiddles(F, log_n, tw, tw_log)) return GSN_OK;
  const int k = std::min(F.max_log_n, std::max(log_n, F.default_tw_log));
  uint32_t r[kMaxLimbs];
  default_root(F, k, r);
  *tw_log = k;
  return powers_table(F, r, k, tw, T, s, /*pin=*/true);
}

int resolve_tables(const FieldOps& F, uint32_t log_n, const uint32_t* omega, int dir, const uint32_t* shift,
                   Tables* T, cudaStream_t stream) {
  T->held.clear();
  if ((int)log_n > F.max_log_n || (int)log_n > F.two_adicity)
    return set_error(GSN_ERR_SIZE, "log_n=%u exceeds the limit %d for field %d", log_n,
                     std::min(F.max_log_n, F.two_adicity), F.id);
  if (dir < GSN_FORWARD || dir > GSN_COSET_INVERSE) return set_error(GSN_ERR_ARG, "bad direction %d", dir);
  const int N = F.limbs;
  uint32_t def[kMaxLimbs];
  default_root(F, (int)log_n, def);
  int rc;
  if (!omega || std::memcmp(omega, def, sizeof(uint32_t) * N) == 0) {
    rc = default_twiddles(F, (int)log_n, &T->tw, &T->tw_log, T, stream);
  } else {
    if (!F.is_canonical(omega)) return set_error(GSN_ERR_OMEGA, "omega is not reduced below the modulus");
    if (!F.is_primitive(omega, (int)log_n))
      return set_error(GSN_ERR_OMEGA, "omega is not a primitive 2^%u-th root of unity", log_n);
    T->tw_log = (int)log_n;
    rc = powers_table(F, omega, (int)log_n, &T->tw, T, stream, T->pin);
  }
  if (rc) return rc;
  std::memcpy(T->root, omega ? omega : def, sizeof(uint32_t) * N);
  T->inverse = (dir == GSN_INVERSE || dir == GSN_COSET_INVERSE) ? 1 : 0;
  T->div_log = T->inverse ? (int)log_n : 0;
  T->pre_table = nullptr;
  T->post_table = nullptr;
  if (dir == GSN_COSET_FORWARD || dir == GSN_COSET_INVERSE) {
    uint32_t s[kMaxLimbs] = {0};
    if (shift) {
      if (!F.is_canonical(shift)) return set_error(GSN_ERR_ARG, "coset shift is not reduced below the modulus");
      std::memcpy(s, shift, sizeof(uint32_t) * N);
    } else {
      s[0] = F.generator;
    }
    bool zero = true;
    for (int i = 0; i < N; ++i) zero = zero && s[i] == 0;
    if (zero) return set_error(GSN_ERR_ARG, "coset shift must be non-zero");
    if (dir == GSN_COSET_FORWARD) {
      rc = powers_table(F, s, (int)log_n, &T->pre_table, T, stream, T->pin);
    } else {
      uint32_t si[kMaxLimbs];
      inv_memo(F, s, si);
      rc = powers_table(F, si, (int)log_n, &T->post_table, T, stream, T->pin);
    }
    if (rc) return rc;
  }
  return GSN_OK;
}

bool find_default_twiddles(const FieldOps& F, int log_n, const uint32_t** tw, int* tw_log) {
  TableCache& C = cache();
  const int dev = current_device();
  std::lock_guard<std::mutex> g(C.mu);
  for (int k = log_n; k <= F.max_log_n; ++k) {
    uint32_t r[kMaxLimbs];
    default_root(F, k, r);
    auto it = C.powers.find(std::make_tuple(dev, F.id, k, limbs_key(r, F.limbs)));
    if (it != C.powers.end()) {
      it->second.pinned = true;  // the caller takes no reference
      *tw = static_cast<const uint32_t*>(it->second.table->p);
      *tw_log = k;
      return true;
    }
  }
  return false;
}

int resolve_p32_tables(const FieldOps& F, const Plan& plan, Tables* T, cudaStream_t s) {
  uint32_t root[kMaxLimbs];
  std::memcpy(root, T->root, sizeof(uint32_t) * F.limbs);
  const int L = plan.log_n;
  if (T->inverse) {
    inv_memo(F, T->root, root);
    uint32_t nn[kMaxLimbs] = {0}, ninv[kMaxLimbs], r[kMaxLimbs];
    nn[0] = 1u << L;  // at most 2^28
    inv_memo(F, nn, ninv);
    F.to_mont(ninv, r);
    T->p32_pre_const = r[0];
  }
  for (int p = 0; p < plan.npass; ++p) {
    const int r = plan.radix_log[p];
    uint32_t wr[kMaxLimbs];
    F.pow(root, (uint64_t)1 << (L - r), wr);  // a primitive 2^r-th root
    int rc = powers_table(F, wr, r - 1, &T->p32_tile[p], T, s, T->pin);
    if (rc) return rc;
  }
  T->p32_lo_bits = (L + 1) / 2;
  int rc = powers_table(F, root, T->p32_lo_bits, &T->p32_lo, T, s, T->pin);
  if (rc) return rc;
  uint32_t hb[kMaxLimbs];
  F.pow(root, (uint64_t)1 << T->p32_lo_bits, hb);
  return powers_table(F, hb, L - T->p32_lo_bits, &T->p32_hi, T, s, T->pin);
}

void full_table_passes(const Plan& plan, Tables* T) {
  for (int p = 0; p < plan.npass; ++p) {
    T->stage[p] = T->tw;
    T->stage_shift[p] = T->tw_log - plan.radix_log[p];
    T->step[p] = nullptr;
  }
}

// Entry k 2^inner + j = w^(j k), w = (root of `tw`)^(2^shift) of order 2^(r + inner), k < 2^r.  r = kStage: entry j = w^j,
// w of order 2^(inner + 1).
constexpr int kStage = -1;
static int pass_table(const FieldOps& F, const uint32_t* tw, int shift, int r, int inner, const std::string& name,
                      const uint32_t** out, PassTables* T) {
  TableCache& C = cache();
  const int dev = current_device();
  std::lock_guard<std::mutex> g(C.mu);
  auto key = std::make_tuple(dev, F.id, r == kStage ? inner + 1 : r + inner, r, name);
  auto it = C.steps.find(key);
  if (it == C.steps.end()) {
    cudaStream_t& gen = C.gen_stream[dev];
    if (!gen) GSN_CUDA(cudaStreamCreateWithFlags(&gen, cudaStreamNonBlocking));
    auto b = std::make_shared<Table>();
    b->bytes = table_words(F, (uint64_t)1 << (r == kStage ? inner : r + inner)) * sizeof(uint32_t);
    const bool room = table_room(C, b->bytes, nullptr);
    t_no_memory = !room;
    int rc = room ? dev_alloc_plain(&b->p, b->bytes)
                  : set_error(GSN_ERR_NOMEM, "held tables take half of the device's memory");
    if (rc) return rc;
    uint32_t* const p = static_cast<uint32_t*>(b->p);
    cudaError_t e = r == kStage ? F.stage_table(p, tw, inner, shift, gen) : F.step_table(p, tw, r, inner, shift, gen);
    if (e == cudaSuccess) e = cudaStreamSynchronize(gen);
    if (e != cudaSuccess) return cuda_fail(e, "pass table");
    count_launches(1);
    b->born = C.births++;
    it = C.steps.emplace(key, b).first;
  }
  T->held.push_back(it->second);
  *out = static_cast<const uint32_t*>(it->second->p);
  return GSN_OK;
}

int resolve_pass_tables(const FieldOps& F, const Plan& plan, Tables* T, cudaStream_t s) {
  full_table_passes(plan, T);
  T->own_passes = true;
  if (F.limbs == 1) return GSN_OK;
  T->own_passes = false;
  TableCache& C = cache();
  const int dev = current_device(), L = plan.log_n;
  std::string tail = limbs_key(T->root, F.limbs);
  for (int p = 0; p < plan.npass; ++p) tail.push_back((char)plan.radix_log[p]);
  const auto key = std::make_tuple(dev, F.id, L, tail);
  std::shared_ptr<const PassTables> found;
  {
    std::lock_guard<std::mutex> g(C.mu);
    auto it = C.passes.find(key);
    if (it != C.passes.end()) found = it->second;
  }
  if (!found || found->stages_only || (found->none && T->pin)) {
    if (capturing(s)) return GSN_OK;
    const bool seen = found != nullptr;
    auto t = std::make_shared<PassTables>();
    uint32_t def[kMaxLimbs];
    default_root(F, L, def);
    std::string name;
    if (std::memcmp(T->root, def, sizeof(uint32_t) * F.limbs) != 0) {
      name = limbs_key(T->root, F.limbs);
      name.push_back((char)L);
    }
    // The factors cost a first call more than they save it, an array's worth of memory to map and to write (BLS12-381 2^20:
    // 577 us in all with them, 411 before there were any), and a program may draw a root for every call.
    t->stages_only = T->single && !seen && !name.empty() && plan.npass > 1;
    int outer = 0, rc = GSN_OK;
    for (int p = 0; p < plan.npass && !rc; ++p) {
      const int r = plan.radix_log[p], left = L - outer;
      if (r >= 1) rc = pass_table(F, T->tw, T->tw_log - r, kStage, r - 1, name, &t->stage[p], t.get());
      if (!rc && p < plan.npass - 1 && !t->stages_only)
        rc = pass_table(F, T->tw, T->tw_log - left, r, left - r, name, &t->step[p], t.get());
      outer += r;
    }
    if (rc == GSN_ERR_NOMEM) {
      if (!t_no_memory) return GSN_OK;
      t = std::make_shared<PassTables>();
      t->none = true;
    } else if (rc) {
      return rc;
    }
    std::lock_guard<std::mutex> g(C.mu);
    t->born = C.births++;
    C.passes[key] = t;
    found = t;
  }
  T->held.push_back(found);
  for (int p = 0; p < plan.npass; ++p) {
    if (found->stage[p]) {
      T->stage[p] = found->stage[p];
      T->stage_shift[p] = 0;
    }
    T->step[p] = found->step[p];
  }
  T->own_passes = !found->stages_only;
  return GSN_OK;
}

uint64_t pass_tables_mark() {
  TableCache& C = cache();
  std::lock_guard<std::mutex> g(C.mu);
  return C.births;
}

void drop_pass_tables_since(uint64_t mark) {
  TableCache& C = cache();
  std::lock_guard<std::mutex> g(C.mu);
  const int dev = current_device();
  if (C.births == mark || cudaDeviceSynchronize() != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  for (auto it = C.passes.begin(); it != C.passes.end();)
    it = std::get<0>(it->first) == dev && it->second->born >= mark && it->second.use_count() == 1 ? C.passes.erase(it)
                                                                                                   : std::next(it);
  for (auto it = C.steps.begin(); it != C.steps.end();)
    it = std::get<0>(it->first) == dev && it->second->born >= mark && it->second.use_count() == 1 ? C.steps.erase(it)
                                                                                                   : std::next(it);
}

int resolve_plan_tables(const FieldOps& F, const Plan& plan, Tables* T, cudaStream_t s) {
  return plan.kernel == kKernelP32 ? resolve_p32_tables(F, plan, T, s) : resolve_pass_tables(F, plan, T, s);
}

int scratch_for(cudaStream_t s, size_t bytes, uint32_t** out, int slot) {
  TableCache& C = cache();
  const int dev = current_device();
  std::lock_guard<std::mutex> g(C.mu);
  DevBuf& b = C.scratch[std::make_tuple(dev, s, slot)];
  if (b.bytes < bytes) {
    if (b.p) {
      GSN_CUDA(cudaStreamSynchronize(s));
      dev_free(b.p);
      b.p = nullptr;
      b.bytes = 0;
    }
    int rc = dev_alloc_locked(C, &b.p, bytes, s);
    if (rc) return rc;
    b.bytes = bytes;
  }
  *out = static_cast<uint32_t*>(b.p);
  return GSN_OK;
}

static size_t scratch_held(cudaStream_t s, int slot) {
  TableCache& C = cache();
  std::lock_guard<std::mutex> g(C.mu);
  const auto it = C.scratch.find(std::make_tuple(current_device(), s, slot));
  return it == C.scratch.end() ? 0 : it->second.bytes;
}

static void pass_arrays(PassArrays* P, bool first, bool last, uint32_t* const* data, uint32_t* const* scratch,
                        int arrays) {
  for (int i = 0; i < arrays; ++i) {
    P->src[i] = first ? data[i] : scratch[i];
    P->dst[i] = last ? data[i] : scratch[i];
  }
}

static int enqueue_p32(const Plan& plan, const Tables& T, uint32_t* const* data, uint32_t* const* scratch, int arrays,
                       cudaStream_t s) {
  const int sms = current_device_sms();
  P32Args A;
  std::memset(&A, 0, sizeof(A));
  A.tw_lo = T.p32_lo;
  A.tw_hi = T.p32_hi;
  A.lo_bits = T.p32_lo_bits;
  A.log_n = plan.log_n;
  A.npass = plan.npass;
  for (int i = 0; i < kMaxPasses; ++i) A.radix_log[i] = plan.radix_log[i];
  int outer = 0;
  for (int p = 0; p < plan.npass; ++p) {
    A.first = p == 0;
    A.last = p == plan.npass - 1;
    pass_arrays(&A.arrays, A.first, A.last, data, scratch, arrays);
    A.tw_tile = T.p32_tile[p];
    A.log_r = plan.radix_log[p];
    A.log_outer = outer;
    A.log_inner = plan.log_n - outer - plan.radix_log[p];
    A.log_j = plan.log_j[p];
    A.tiles = (uint64_t)1 << (plan.log_n - A.log_r - A.log_j);
    A.pre_table = A.first ? T.pre_table : nullptr;
    A.post_table = A.last ? T.post_table : nullptr;
    A.has_pre_const = A.first ? T.inverse : 0;
    A.pre_const = T.p32_pre_const;
    cudaError_t e = launch_p32_pass(A, arrays, plan.e_log, plan.block[p], sms * 16, s);
    if (e != cudaSuccess) return cuda_fail(e, "p32 NTT pass launch");
    count_launches(1);
    outer += plan.radix_log[p];
  }
  return GSN_OK;
}

int load_plan(const FieldOps& F, const Plan& plan) {
  cudaError_t e = plan.kernel == kKernelLanes ? F.load_lanes() : F.load();
  if (plan.kernel == kKernelP32) {
    P32Args A;
    std::memset(&A, 0, sizeof(A));
    for (int p = 0; p < plan.npass && e == cudaSuccess; ++p) {
      A.last = p == plan.npass - 1;
      A.log_r = plan.radix_log[p];
      A.log_j = plan.log_j[p];
      e = launch_p32_pass(A, /*arrays=*/0, plan.e_log, plan.block[p], 1, nullptr);
    }
  }
  return e == cudaSuccess ? GSN_OK : cuda_fail(e, "kernel load");
}

int enqueue_ntt(const FieldOps& F, const Plan& plan, const Tables& T, uint32_t* data, uint32_t* scratch,
                cudaStream_t s) {
  return enqueue_ntts(F, plan, T, &data, &scratch, 1, s);
}

int enqueue_ntts(const FieldOps& F, const Plan& plan, const Tables& T, uint32_t* const* data, uint32_t* const* scratch,
                 int arrays, cudaStream_t s) {
  if (plan.kernel == kKernelP32) return enqueue_p32(plan, T, data, scratch, arrays, s);
  const bool lanes = plan.kernel == kKernelLanes;
  PassArgs A;
  std::memset(&A, 0, sizeof(A));
  A.tw = T.tw;
  A.tw_log = T.tw_log;
  A.log_n = plan.log_n;
  A.inverse = T.inverse;
  A.npass = plan.npass;
  for (int i = 0; i < kMaxPasses; ++i) A.radix_log[i] = plan.radix_log[i];
  int outer = 0;
  for (int p = 0; p < plan.npass; ++p) {
    A.first = p == 0;
    A.last = p == plan.npass - 1;
    pass_arrays(&A.arrays, A.first, A.last, data, scratch, arrays);
    A.log_r = plan.radix_log[p];
    A.log_outer = outer;
    A.log_inner = plan.log_n - outer - plan.radix_log[p];
    A.log_j = plan.log_j[p];
    A.tiles = (uint64_t)1 << (plan.log_n - A.log_r - A.log_j);
    A.stage_tw = T.stage[p];
    A.stage_shift = T.stage_shift[p];
    A.step_tw = T.step[p];
    A.pre_table = A.first ? T.pre_table : nullptr;
    A.post_table = A.last ? T.post_table : nullptr;
    A.div_log = A.last ? T.div_log : 0;
    cudaError_t e = lanes ? F.pass_lanes(A, arrays, plan.block[p], s) : F.pass(A, arrays, plan.block[p], s);
    if (e != cudaSuccess) return cuda_fail(e, "NTT pass launch");
    count_launches(1);
    outer += plan.radix_log[p];
  }
  return GSN_OK;
}

static int check_data_ptr(const FieldOps& F, const void* p) {
  if (!p) return set_error(GSN_ERR_ARG, "null data pointer");
  const uintptr_t align = (F.limbs % 4 == 0) ? 16 : 4;
  if (reinterpret_cast<uintptr_t>(p) % align)
    return set_error(GSN_ERR_ARG, "data pointer must be %zu-byte aligned", (size_t)align);
  return GSN_OK;
}

// What a transform call resolves to, by the values of its arguments.  Resolving takes a look-up per table, and for a
// caller's own root the test that it is primitive (2^log_n-fold squaring on the host: 72 us for 24 limbs and 2^18);
// small transforms take 10 us on the GPU.  Dropped when a plan changes or the caches are released.
struct Call {
  Plan plan;
  Tables tables;
};
struct Calls {
  std::mutex mu;
  uint64_t generation = 0;
  // (device, field, log_n, direction, 16-byte aligned, within a QAP computation, omega limbs, shift limbs; empty
  // strings for the defaults)
  std::map<std::tuple<int, int, uint32_t, int, bool, bool, std::string, std::string>, std::shared_ptr<const Call>> known;
};
constexpr size_t kMaxCalls = 4096;  // about 1 KB each; the tables they hold are given back when memory runs out
static Calls& calls() {
  static Calls* c = new Calls();
  return *c;
}
static void forget_calls() {
  Calls& K = calls();
  std::lock_guard<std::mutex> g(K.mu);
  ++K.generation;
  K.known.clear();
}

// Four lanes per product pay while the chip is not full, and a kernel's code has to be fetched anew when others run
// between its launches. QAP computations on GB300, lanes against a thread per product: 2^12 144 and 163 us, 2^13 217 and
// 179 (206 with lanes in the last, single transform alone).
constexpr uint32_t kLanesMaxLogQap = 12;

// ptrs: the arrays, and the caller's scratch, whose alignment counts; qap: a step of a QAP computation.
static int resolve_call(const FieldOps& F, uint32_t log_n, const uint32_t* omega, int dir, const uint32_t* shift,
                        const void* const* ptrs, int count, bool qap, cudaStream_t s,
                        std::shared_ptr<const Call>* out) {
  bool aligned = true;  // the multi-limb fields' arrays always are
  for (int i = 0; i < count; ++i) aligned = aligned && reinterpret_cast<uintptr_t>(ptrs[i]) % 16 == 0;
  const auto key = std::make_tuple(current_device(), F.id, log_n, dir, aligned, qap,
                                   omega ? limbs_key(omega, F.limbs) : std::string(),
                                   shift ? limbs_key(shift, F.limbs) : std::string());
  Calls& K = calls();
  uint64_t generation;
  {
    std::lock_guard<std::mutex> g(K.mu);
    const auto it = K.known.find(key);
    if (it != K.known.end()) {
      *out = it->second;
      return GSN_OK;
    }
    generation = K.generation;
  }
  auto call = std::make_shared<Call>();
  call->tables.single = true;
  int rc = resolve_tables(F, log_n, omega, dir, shift, &call->tables, s);
  if (rc) return rc;
  call->plan = plan_for(F, (int)log_n);
  if (call->plan.kernel == kKernelP32 && !aligned) {
    // the register-blocked 32-bit pass moves 16-byte vectors; 4-byte-aligned arrays take the generic pass
    const FieldLimits L = limits_of(F);
    call->plan = make_plan(F, (int)log_n, L.max_r, L.target_j, L.max_block);
  }
  if (call->plan.kernel == kKernelLanes && qap && log_n > kLanesMaxLogQap) {
    // two near-equal passes, or more where a radix would pass the field's usual limit (2^12 does not fit shared memory)
    const int npass = std::max(2, ((int)log_n + limits_of(F).max_r - 1) / limits_of(F).max_r);
    int radix[kMaxPasses] = {0, 0, 0, 0};
    for (int i = 0; i < npass; ++i) radix[i] = (int)log_n * (i + 1) / npass - (int)log_n * i / npass;
    call->plan = make_split_plan(F, (int)log_n, radix, npass, /*target_j=*/0, 128);
  }
  rc = resolve_plan_tables(F, call->plan, &call->tables, s);
  if (rc) return rc;
  *out = call;
  if (call->plan.kernel == kKernelP32 || call->tables.own_passes) {
    std::lock_guard<std::mutex> g(K.mu);
    if (K.known.size() >= kMaxCalls) K.known.clear();  // a shift drawn anew for every call
    if (K.generation == generation) K.known.emplace(key, call);
  }
  return GSN_OK;
}

// A captured call's tables stay as long as its graph may run.
static void hold_captured(const std::shared_ptr<const Call>& call, cudaStream_t s) {
  if (!capturing(s)) return;
  TableCache& C = cache();
  std::lock_guard<std::mutex> g(C.mu);
  C.captured.insert(call);
}

static int ntt_impl(int field, uint32_t* data, uint32_t log_n, const uint32_t* omega, int dir,
                    const uint32_t* shift, uint32_t* scratch, cudaStream_t s, bool qap = false) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  int rc = check_data_ptr(*F, data);
  if (rc) return rc;
  if (scratch) {
    rc = check_data_ptr(*F, scratch);
    if (rc) return rc;
  }
  std::shared_ptr<const Call> call;
  const void* const ptrs[2] = {data, scratch};
  rc = resolve_call(*F, log_n, omega, dir, shift, ptrs, 2, qap, s, &call);
  if (rc) return rc;
  const Plan& plan = call->plan;
  hold_captured(call, s);
  if (plan.npass > 1 && !scratch) {
    rc = scratch_for(s, ((size_t)1 << log_n) * F->limbs * sizeof(uint32_t), &scratch);
    if (rc) return rc;
  }
  return enqueue_ntt(*F, plan, call->tables, data, scratch, s);
}

// zr2 = z * R^2 with z = 1 / Z(shift * w^i) = 1 / (shift^n - 1), the inverse vanishing polynomial of the
// size-n radix-2 domain on its coset by `shift` (null: the field's generator).
static int coset_z_inv(const FieldOps& F, uint32_t log_n, const uint32_t* shift, uint32_t* zr2) {
  uint32_t s[kMaxLimbs] = {0}, t[kMaxLimbs] = {0}, u[kMaxLimbs] = {0};
  if (shift) {
    if (!F.is_canonical(shift)) return set_error(GSN_ERR_ARG, "shift is not a canonical field element");
    std::memcpy(s, shift, F.limbs * sizeof(uint32_t));
  } else {
    s[0] = F.generator;
  }
  bool zero = true;
  for (int i = 0; i < F.limbs; ++i) zero = zero && s[i] == 0;
  if (zero) return set_error(GSN_ERR_ARG, "shift must be nonzero");
  F.pow(s, (uint64_t)1 << log_n, t);
  bool one = t[0] == 1;
  for (int i = 1; i < F.limbs; ++i) one = one && t[i] == 0;
  if (one) return set_error(GSN_ERR_ARG, "shift^n = 1: Z(x) = x^n - 1 vanishes on that coset");
  for (int i = 0; i < F.limbs; ++i) {  // t - 1; t >= 2 here
    if (t[i]--) break;
  }
  inv_memo(F, t, u);
  F.to_mont(u, t);
  F.to_mont(t, zr2);
  return GSN_OK;
}

static int quotient_impl(int field, uint32_t* a, const uint32_t* b, const uint32_t* c, uint32_t log_n,
                         const uint32_t* shift, cudaStream_t s) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  if ((int)log_n > F->two_adicity) return set_error(GSN_ERR_SIZE, "log_n=%u exceeds the 2-adicity", log_n);
  int rc = check_data_ptr(*F, a);
  if (!rc) rc = check_data_ptr(*F, b);
  if (!rc) rc = check_data_ptr(*F, c);
  if (rc) return rc;
  uint32_t zr2[kMaxLimbs];
  rc = coset_z_inv(*F, log_n, shift, zr2);
  if (rc) return rc;
  cudaError_t e = F->quotient(a, b, c, (uint64_t)1 << log_n, zr2, s);
  if (e != cudaSuccess) return cuda_fail(e, "coset quotient launch");
  count_launches(1);
  return GSN_OK;
}

// The three polynomials of a QAP computation go through their transforms in the same launches while they and their
// scratch stay in half of the 129 MB L2.  A pass on one small array leaves most of the chip idle.
static bool qap_together(const FieldOps& F, uint32_t log_n) {
  return log_n < 32 && (((uint64_t)2 * kMaxArrays * F.limbs * sizeof(uint32_t)) << log_n) <= ((uint64_t)64 << 20);
}

// Inverse, then coset transform of three arrays.  GSN_ERR_NOMEM, before anything is enqueued, if there is no memory for
// three arrays of scratch or for a table.
static int qap_arrays(const FieldOps& F, uint32_t* const* polys, uint32_t log_n, const uint32_t* shift,
                      cudaStream_t s) {
  for (int i = 0; i < kMaxArrays; ++i) {
    int rc = check_data_ptr(F, polys[i]);
    if (rc) return rc;
  }
  const void* const ptrs[kMaxArrays] = {polys[0], polys[1], polys[2]};
  std::shared_ptr<const Call> inv, fwd;
  int rc = resolve_call(F, log_n, nullptr, GSN_INVERSE, nullptr, ptrs, kMaxArrays, true, s, &inv);
  if (!rc) rc = resolve_call(F, log_n, nullptr, GSN_COSET_FORWARD, shift, ptrs, kMaxArrays, true, s, &fwd);
  if (rc) return rc;
  // One array's scratch is a transform's own, so that no buffer a captured transform holds grows here; the others' lie
  // in a buffer beside it.
  const size_t one = ((size_t)F.limbs << log_n) * sizeof(uint32_t);
  const size_t step = (one + 15) & ~(size_t)15, others = (kMaxArrays - 1) * step;  // 16-byte aligned
  uint32_t* scratch[kMaxArrays] = {nullptr, nullptr, nullptr};
  if (std::max(inv->plan.npass, fwd->plan.npass) > 1) {
    // growing a buffer would end a capture
    if (capturing(s) && (scratch_held(s, 0) < one || scratch_held(s, kScratchArrays) < others)) return GSN_ERR_NOMEM;
    rc = scratch_for(s, one, &scratch[0]);
    if (!rc) rc = scratch_for(s, others, &scratch[1], kScratchArrays);
    if (rc) return rc;
    for (int i = 2; i < kMaxArrays; ++i) scratch[i] = scratch[1] + (i - 1) * (step / sizeof(uint32_t));
  }
  hold_captured(inv, s);
  hold_captured(fwd, s);
  rc = enqueue_ntts(F, inv->plan, inv->tables, polys, scratch, kMaxArrays, s);
  return rc ? rc : enqueue_ntts(F, fwd->plan, fwd->tables, polys, scratch, kMaxArrays, s);
}

// Device buffers, streams and events of the host-memory entry points (gsn_ntt_host, gsn_ntt_host_batch).  A
// call checks one state out of an idle pool for the current device (or makes a new one) and returns it when
// done, so concurrent callers on different host threads each run on their own buffers and streams and none
// waits for another.  gsn_release_caches frees the idle states.
struct HostState {
  static constexpr int kBufs = 3;
  int dev = 0;
  cudaStream_t s_in = nullptr, s_comp = nullptr, s_out = nullptr;
  cudaEvent_t ev_in[kBufs] = {}, ev_comp[kBufs] = {}, ev_out[kBufs] = {};
  DevBuf bufs[kBufs];
};

static std::mutex g_host_pool_mu;
static std::vector<HostState*> g_host_idle;

static void host_state_destroy(HostState* h) {
  for (DevBuf& b : h->bufs) dev_free(b.p);
  for (cudaStream_t s : {h->s_in, h->s_comp, h->s_out})
    if (s) cudaStreamDestroy(s);
  for (int b = 0; b < HostState::kBufs; ++b)
    for (cudaEvent_t e : {h->ev_in[b], h->ev_comp[b], h->ev_out[b]})
      if (e) cudaEventDestroy(e);
  delete h;
}

static int host_state_acquire(HostState** out) {
  const int dev = current_device();
  {
    std::lock_guard<std::mutex> g(g_host_pool_mu);
    for (size_t i = 0; i < g_host_idle.size(); ++i) {
      if (g_host_idle[i]->dev == dev) {
        *out = g_host_idle[i];
        g_host_idle.erase(g_host_idle.begin() + (long)i);
        return GSN_OK;
      }
    }
  }
  HostState* h = new HostState();
  h->dev = dev;
  cudaError_t e = cudaSuccess;
  for (cudaStream_t* s : {&h->s_in, &h->s_comp, &h->s_out})
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(s, cudaStreamNonBlocking);
  for (int b = 0; b < HostState::kBufs && e == cudaSuccess; ++b)
    for (cudaEvent_t* ev : {&h->ev_in[b], &h->ev_comp[b], &h->ev_out[b]})
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    host_state_destroy(h);
    return cuda_fail(e, "host-path stream and event creation");
  }
  *out = h;
  return GSN_OK;
}

static void host_state_release(HostState* h) {
  std::lock_guard<std::mutex> g(g_host_pool_mu);
  g_host_idle.push_back(h);
}

// Grows buffer k of a checked-out state to `bytes` (after the state's streams have drained).
static int host_state_buffer(HostState* h, int k, size_t bytes) {
  DevBuf& b = h->bufs[k];
  if (b.bytes >= bytes) return GSN_OK;
  GSN_CUDA(cudaStreamSynchronize(h->s_out));
  GSN_CUDA(cudaStreamSynchronize(h->s_comp));
  dev_free(b.p);
  b.p = nullptr;
  b.bytes = 0;
  int rc = dev_alloc(&b.p, bytes);
  if (rc) return rc;
  b.bytes = bytes;
  return GSN_OK;
}
}  // namespace gsn

using namespace gsn;

extern "C" {

const char* gsn_last_error(void) { return t_error.c_str(); }

int gsn_version(void) { return 100; }

int gsn_field_limbs(int field) {
  const FieldOps* F = field_ops(field);
  return F ? F->limbs : -GSN_ERR_FIELD;
}

int gsn_field_two_adicity(int field) {
  const FieldOps* F = field_ops(field);
  return F ? F->two_adicity : -GSN_ERR_FIELD;
}

int gsn_field_max_log_n(int field) {
  const FieldOps* F = field_ops(field);
  return F ? std::min(F->max_log_n, F->two_adicity) : -GSN_ERR_FIELD;
}

int gsn_field_modulus(int field, uint32_t* out) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  if (!out) return set_error(GSN_ERR_ARG, "null output");
  F->modulus(out);
  return GSN_OK;
}

int gsn_root_of_unity(int field, uint32_t log_n, uint32_t* out) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  if (!out) return set_error(GSN_ERR_ARG, "null output");
  if ((int)log_n > F->two_adicity) return set_error(GSN_ERR_SIZE, "log_n exceeds the 2-adicity");
  F->root((int)log_n, out);
  return GSN_OK;
}

int gsn_ntt(int field, uint32_t* data, uint32_t log_n, const uint32_t* omega, int dir, const uint32_t* shift,
            void* stream) {
  return ntt_impl(field, data, log_n, omega, dir, shift, nullptr, static_cast<cudaStream_t>(stream));
}

int gsn_ntt_scratch(int field, uint32_t* data, uint32_t log_n, const uint32_t* omega, int dir,
                    const uint32_t* shift, uint32_t* scratch, void* stream) {
  if (!scratch) return set_error(GSN_ERR_ARG, "null scratch");
  return ntt_impl(field, data, log_n, omega, dir, shift, scratch, static_cast<cudaStream_t>(stream));
}

int gsn_ntt_host(int field, uint32_t* data, uint32_t log_n, const uint32_t* omega, int dir,
                 const uint32_t* shift) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  if (!data) return set_error(GSN_ERR_ARG, "null data pointer");
  if ((int)log_n > std::min(F->max_log_n, F->two_adicity))
    return set_error(GSN_ERR_SIZE, "log_n=%u exceeds the limit for field %d", log_n, field);
  HostState* h = nullptr;
  int rc = host_state_acquire(&h);
  if (rc) return rc;
  const size_t bytes = ((size_t)1 << log_n) * F->limbs * sizeof(uint32_t);
  rc = host_state_buffer(h, 0, bytes);
  if (!rc) {
    uint32_t* dev = static_cast<uint32_t*>(h->bufs[0].p);
    const cudaStream_t stream = h->s_comp;
    cudaError_t e = cudaMemcpyAsync(dev, data, bytes, cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) rc = cuda_fail(e, "host-to-device copy");
    if (!rc) rc = ntt_impl(field, dev, log_n, omega, dir, shift, nullptr, stream);
    if (!rc) {
      e = cudaMemcpyAsync(data, dev, bytes, cudaMemcpyDeviceToHost, stream);
      if (e != cudaSuccess) rc = cuda_fail(e, "device-to-host copy");
    }
    e = cudaStreamSynchronize(stream);
    if (!rc && e != cudaSuccess) rc = cuda_fail(e, "cudaStreamSynchronize");
  }
  host_state_release(h);
  return rc;
}

// Copies of array i+1 (in) and i-1 (out) overlap the transform of array i: three device buffers in
// rotation, copy-in, transform and copy-out on their own streams, ordered by events.
static int host_batch_run(HostState* h, const FieldOps* F, int field, uint32_t* const* data, size_t count,
                          uint32_t log_n, const uint32_t* omega, int dir, const uint32_t* shift) {
  constexpr int kBufs = HostState::kBufs;
  const size_t bytes = ((size_t)1 << log_n) * F->limbs * sizeof(uint32_t);
  for (int k = 0; k < kBufs; ++k) {
    int rc = host_state_buffer(h, k, bytes);
    if (rc) return rc;
  }
  for (size_t i = 0; i < count; ++i) {
    const int b = (int)(i % kBufs);
    uint32_t* dev = static_cast<uint32_t*>(h->bufs[b].p);
    if (i >= kBufs) GSN_CUDA(cudaStreamWaitEvent(h->s_in, h->ev_out[b], 0));  // array i-3 has left this buffer
    GSN_CUDA(cudaMemcpyAsync(dev, data[i], bytes, cudaMemcpyHostToDevice, h->s_in));
    GSN_CUDA(cudaEventRecord(h->ev_in[b], h->s_in));
    GSN_CUDA(cudaStreamWaitEvent(h->s_comp, h->ev_in[b], 0));
    int rc = ntt_impl(field, dev, log_n, omega, dir, shift, nullptr, h->s_comp);
    if (rc) return rc;
    GSN_CUDA(cudaEventRecord(h->ev_comp[b], h->s_comp));
    GSN_CUDA(cudaStreamWaitEvent(h->s_out, h->ev_comp[b], 0));
    GSN_CUDA(cudaMemcpyAsync(data[i], dev, bytes, cudaMemcpyDeviceToHost, h->s_out));
    GSN_CUDA(cudaEventRecord(h->ev_out[b], h->s_out));
  }
  return GSN_OK;
}

int gsn_ntt_host_batch(int field, uint32_t* const* data, size_t count, uint32_t log_n, const uint32_t* omega,
                       int dir, const uint32_t* shift) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  if (count && !data) return set_error(GSN_ERR_ARG, "null array list");
  for (size_t i = 0; i < count; ++i)
    if (!data[i]) return set_error(GSN_ERR_ARG, "null data pointer at %zu", i);
  if ((int)log_n > std::min(F->max_log_n, F->two_adicity))
    return set_error(GSN_ERR_SIZE, "log_n=%u exceeds the limit for field %d", log_n, field);
  if (count == 0) return GSN_OK;
  HostState* h = nullptr;
  int rc = host_state_acquire(&h);
  if (rc) return rc;
  rc = host_batch_run(h, F, field, data, count, log_n, omega, dir, shift);
  // drain all three streams, also after a failure, before the state goes back to the pool
  for (cudaStream_t s : {h->s_in, h->s_comp, h->s_out}) {
    cudaError_t e = cudaStreamSynchronize(s);
    if (!rc && e != cudaSuccess) rc = cuda_fail(e, "cudaStreamSynchronize");
  }
  host_state_release(h);
  return rc;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// multi-exponentiation over field elements (cuda/multi_exp.cu:104-137, test/multiexp.h:3-13)
// ---------------------------------------------------------------------------
namespace gsn {
// The representation constant of multiexp.cuh: 2^(32(2N+2)) mod p (canonical) or 2^(32(N+2)) mod p
// (Montgomery), canonical limbs.  Computed once per (field, mode): the host exponentiation takes longer
// than a whole small multi-exponentiation on the GPU.
static void multiexp_fix(const FieldOps& F, int mode, uint32_t* fix) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, std::string> memo;
  std::lock_guard<std::mutex> g(mu);
  auto key = std::make_pair(F.id, mode);
  auto it = memo.find(key);
  if (it == memo.end()) {
    uint32_t two[kMaxLimbs] = {0}, r[kMaxLimbs] = {0};
    two[0] = 2;
    const int N = F.limbs;
    F.pow(two, (uint64_t)32 * (mode == GSN_MULTIEXP_CANONICAL ? 2 * N + 2 : N + 2), r);
    it = memo.emplace(key, limbs_key(r, N)).first;
  }
  std::memcpy(fix, it->second.data(), it->second.size());
}

// Scratch for the blocks' column sums.  A transform's buffer is not grown for them, since a captured transform may hold
// it: they take a buffer of their own, or, while `s` is captured, as few blocks as fit.
static int multiexp_scratch(const FieldOps& F, cudaStream_t s, int* grid, uint32_t** out) {
  const size_t need = F.multiexp_bytes(*grid), block = F.multiexp_bytes(1), held = scratch_held(s, 0);
  if (scratch_held(s, kScratchSums) >= need) return scratch_for(s, need, out, kScratchSums);
  if (held >= need || held == 0) return scratch_for(s, need, out);
  if (held < block || !capturing(s)) return scratch_for(s, need, out, kScratchSums);
  *grid = (int)(held / block);
  return scratch_for(s, held, out);
}

static int multiexp_impl(const FieldOps& F, const uint32_t* a, const uint32_t* b, uint64_t n, uint32_t* out,
                         int mode, cudaStream_t s) {
  int grid = F.multiexp_grid(n);
  uint32_t* partial = nullptr;
  int rc = multiexp_scratch(F, s, &grid, &partial);
  if (rc) return rc;
  uint32_t fix[kMaxLimbs];
  multiexp_fix(F, mode, fix);
  cudaError_t e = F.multiexp(a, b, n, partial, grid, out, fix, s);
  if (e != cudaSuccess) return cuda_fail(e, "multiexp launch");
  count_launches(2);
  return GSN_OK;
}

// Arguments shared by the device and host entry points.
static int multiexp_check(const FieldOps* F, int field, const void* a, const void* b, uint64_t n, const void* out,
                          int mode) {
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  if (mode != GSN_MULTIEXP_CANONICAL && mode != GSN_MULTIEXP_MONTGOMERY)
    return set_error(GSN_ERR_ARG, "bad multiexp mode %d", mode);
  if (!out) return set_error(GSN_ERR_ARG, "null output");
  if (n && (!a || !b)) return set_error(GSN_ERR_ARG, "null input array");
  // each thread adds fewer than 2^32 products to its 2N+1 words, and the total stays below p * 2^(32(N+2))
  if (n > ((uint64_t)1 << 40)) return set_error(GSN_ERR_SIZE, "n = %llu exceeds 2^40", (unsigned long long)n);
  return GSN_OK;
}
}  // namespace gsn

extern "C" {

int gsn_multiexp(int field, const uint32_t* a, const uint32_t* b, uint64_t n, uint32_t* out, int mode,
                 void* stream) {
  const FieldOps* F = field_ops(field);
  int rc = multiexp_check(F, field, a, b, n, out, mode);
  if (rc) return rc;
  const uintptr_t align = (F->limbs % 4 == 0) ? 16 : 4;
  if ((reinterpret_cast<uintptr_t>(out) % align) ||
      (n && ((reinterpret_cast<uintptr_t>(a) % align) || (reinterpret_cast<uintptr_t>(b) % align))))
    return set_error(GSN_ERR_ARG, "a, b and out must be %zu-byte aligned", (size_t)align);
  return multiexp_impl(*F, a, b, n, out, mode, static_cast<cudaStream_t>(stream));
}

int gsn_multiexp_host(int field, const uint32_t* a, const uint32_t* b, uint64_t n, uint32_t* out, int mode) {
  const FieldOps* F = field_ops(field);
  int rc = multiexp_check(F, field, a, b, n, out, mode);
  if (rc) return rc;
  HostState* h = nullptr;
  rc = host_state_acquire(&h);
  if (rc) return rc;
  const size_t bytes = (size_t)n * F->limbs * sizeof(uint32_t), rbytes = F->limbs * sizeof(uint32_t);
  rc = host_state_buffer(h, 0, bytes);
  if (!rc) rc = host_state_buffer(h, 1, bytes);
  if (!rc) rc = host_state_buffer(h, 2, rbytes);
  if (!rc) {
    const cudaStream_t s = h->s_comp;
    uint32_t* da = static_cast<uint32_t*>(h->bufs[0].p);
    uint32_t* db = static_cast<uint32_t*>(h->bufs[1].p);
    uint32_t* dout = static_cast<uint32_t*>(h->bufs[2].p);
    cudaError_t e = cudaSuccess;
    if (bytes) e = cudaMemcpyAsync(da, a, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && bytes) e = cudaMemcpyAsync(db, b, bytes, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) rc = cuda_fail(e, "host-to-device copy");
    if (!rc) rc = multiexp_impl(*F, da, db, n, dout, mode, s);
    if (!rc) {
      e = cudaMemcpyAsync(out, dout, rbytes, cudaMemcpyDeviceToHost, s);
      if (e != cudaSuccess) rc = cuda_fail(e, "device-to-host copy");
    }
    e = cudaStreamSynchronize(s);
    if (!rc && e != cudaSuccess) rc = cuda_fail(e, "cudaStreamSynchronize");
  }
  host_state_release(h);
  return rc;
}

}  // extern "C"

extern "C" {

int gsn_prepare(int field, uint32_t log_n, const uint32_t* omega) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  Tables T;
  T.pin = true;
  int rc = resolve_tables(*F, log_n, omega, GSN_FORWARD, nullptr, &T, nullptr);
  if (rc || F->limbs == 1) return rc;
  return resolve_pass_tables(*F, plan_for(*F, (int)log_n), &T, nullptr);
}

int gsn_pointwise_mul(int field, uint32_t* a, const uint32_t* b, uint64_t n, void* stream) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  int rc = check_data_ptr(*F, a);
  if (rc) return rc;
  rc = check_data_ptr(*F, b);
  if (rc) return rc;
  if (n == 0) return GSN_OK;
  cudaError_t e = F->pointwise(a, b, n, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return cuda_fail(e, "pointwise multiply launch");
  count_launches(1);
  return GSN_OK;
}

int gsn_coset_quotient(int field, uint32_t* a, const uint32_t* b, const uint32_t* c, uint32_t log_n,
                       const uint32_t* shift, void* stream) {
  return quotient_impl(field, a, b, c, log_n, shift, static_cast<cudaStream_t>(stream));
}

int gsn_qap_h(int field, uint32_t* a, uint32_t* b, uint32_t* c, uint32_t log_n, const uint32_t* shift,
              void* stream) {
  if (!a || !b || !c) return set_error(GSN_ERR_ARG, "null data pointer");
  if (a == b || a == c || b == c) return set_error(GSN_ERR_ARG, "a, b and c must be distinct arrays");
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  uint32_t* polys[3] = {a, b, c};
  // evaluations on the domain -> coefficients -> evaluations on the coset
  const FieldOps* F = field_ops(field);
  int rc = F && qap_together(*F, log_n) ? qap_arrays(*F, polys, log_n, shift, s) : GSN_ERR_NOMEM;
  if (rc == GSN_ERR_NOMEM) {
    for (uint32_t* x : polys) {
      rc = ntt_impl(field, x, log_n, nullptr, GSN_INVERSE, nullptr, nullptr, s);
      if (!rc) rc = ntt_impl(field, x, log_n, nullptr, GSN_COSET_FORWARD, shift, nullptr, s);
      if (rc) return rc;
    }
  }
  if (rc) return rc;
  rc = quotient_impl(field, a, b, c, log_n, shift, s);
  if (rc) return rc;
  return ntt_impl(field, a, log_n, nullptr, GSN_COSET_INVERSE, shift, nullptr, s, /*qap=*/true);
}

int gsn_convert(int field, uint32_t* data, uint64_t n, int mode, void* stream) {
  const FieldOps* F = field_ops(field);
  if (!F) return set_error(GSN_ERR_FIELD, "unknown field %d", field);
  if (mode < GSN_TO_MONTGOMERY || mode > GSN_REVERSE_LIMBS) return set_error(GSN_ERR_ARG, "bad mode %d", mode);
  int rc = check_data_ptr(*F, data);
  if (rc) return rc;
  if (n == 0) return GSN_OK;
  cudaError_t e = F->convert(data, n, mode, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return cuda_fail(e, "convert launch");
  count_launches(1);
  return GSN_OK;
}

int gsn_synchronize(void* stream) {
  GSN_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  return GSN_OK;
}

int gsn_host_alloc(void** ptr, size_t bytes) {
  if (!ptr) return set_error(GSN_ERR_ARG, "null output");
  cudaError_t e = cudaMallocHost(ptr, bytes ? bytes : 16);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_error(GSN_ERR_NOMEM, "cudaMallocHost(%zu) failed: %s", bytes, cudaGetErrorString(e));
  }
  return GSN_OK;
}

int gsn_host_free(void* ptr) {
  if (ptr) GSN_CUDA(cudaFreeHost(ptr));
  return GSN_OK;
}

int gsn_release_caches(void) {
  GSN_CUDA(cudaDeviceSynchronize());
  forget_calls();
  {
    std::lock_guard<std::mutex> gh(g_host_pool_mu);
    for (HostState* h : g_host_idle) host_state_destroy(h);
    g_host_idle.clear();
  }
  TableCache& C = cache();
  std::lock_guard<std::mutex> g(C.mu);
  C.captured.clear();
  C.passes.clear();
  C.steps.clear();
  C.powers.clear();
  for (auto& kv : C.scratch) dev_free(kv.second.p);
  C.scratch.clear();
  return GSN_OK;
}

uint64_t gsn_kernel_launch_count(void) { return g_launches.load(); }

}  // extern "C"
