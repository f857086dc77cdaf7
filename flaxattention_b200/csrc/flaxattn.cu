// Host side of the C ABI declared in include/flaxattn.h, plus the kernels that do not
// depend on a score_mod / mask_mod (table compaction, backward preprocess, decode combine).
//
// Kernels that embed user mods are compiled at run time: the mod fragment is placed in
// front of a kernel template from the kernels/ directory, compiled for sm_100a with
// NVRTC, cached in memory per module and on disk per content hash, and loaded through the
// context-independent library API of the CUDA runtime.
#include <cuda_runtime.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <nvrtc.h>

#include <dlfcn.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <map>
#include <mutex>
#include <sstream>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/flaxattn.h"
#include "kernels/fa_params.h"

#ifndef FA_STATIC_SCRATCH_BYTES
#define FA_STATIC_SCRATCH_BYTES (16u << 20)
#endif
constexpr size_t kStaticScratchBytes = (size_t)FA_STATIC_SCRATCH_BYTES;

namespace {

thread_local std::string g_err;
int fail(int code, const std::string& msg) {
  g_err = msg;
  return code;
}
#define FA_CUDA_CHECK(expr)                                                                       \
  do {                                                                                            \
    cudaError_t e_ = (expr);                                                                      \
    if (e_ != cudaSuccess)                                                                        \
      return fail(FA_ECUDA, std::string(#expr) + ": " + cudaGetErrorName(e_) + ": " + cudaGetErrorString(e_)); \
  } while (0)

std::mutex g_mu;
std::string g_kernel_dir, g_cache_dir;
bool g_cache_dir_set = false;
std::atomic<int> g_compile_count{0};

// ---- small utilities -------------------------------------------------------------------
uint64_t fnv1a(const std::string& s, uint64_t seed) {
  uint64_t h = seed;
  for (unsigned char c : s) {
    h ^= c;
    h *= 1099511628211ull;
  }
  return h;
}
std::string hash_hex(const std::string& s) {
  char buf[40];
  snprintf(buf, sizeof buf, "%016llx%016llx", (unsigned long long)fnv1a(s, 1469598103934665603ull),
           (unsigned long long)fnv1a(s, 0x9e3779b97f4a7c15ull));
  return buf;
}
bool read_file(const std::string& path, std::string& out) {
  std::ifstream f(path, std::ios::binary);
  if (!f) return false;
  std::ostringstream ss;
  ss << f.rdbuf();
  out = ss.str();
  return true;
}
void mkdirs(const std::string& path) {
  std::string cur;
  for (size_t i = 0; i < path.size(); ++i) {
    cur.push_back(path[i]);
    if (path[i] == '/' || i + 1 == path.size()) mkdir(cur.c_str(), 0755);
  }
}
std::string kernel_dir() {
  if (!g_kernel_dir.empty()) return g_kernel_dir;
  if (const char* e = getenv("FLAXATTN_KERNEL_DIR")) return g_kernel_dir = e;
  Dl_info info;
  if (dladdr((void*)&fnv1a, &info) && info.dli_fname) {
    std::string p = info.dli_fname;
    size_t k = p.rfind('/');
    const std::string base = k == std::string::npos ? std::string(".") : p.substr(0, k);
    struct stat sb;
    g_kernel_dir = base + "/kernels";
    if (stat(g_kernel_dir.c_str(), &sb) != 0) g_kernel_dir = base + "/csrc/kernels";
  } else {
    g_kernel_dir = "kernels";
  }
  return g_kernel_dir;
}
std::string cache_dir() {
  if (g_cache_dir_set) return g_cache_dir;
  g_cache_dir_set = true;
  if (const char* e = getenv("FLAXATTN_CACHE_DIR")) return g_cache_dir = e;
  const char* home = getenv("HOME");
  g_cache_dir = std::string(home ? home : "/tmp") + "/.cache/flaxattn_b200";
  return g_cache_dir;
}

const char* const kTemplateFiles[] = {"fa_params.h", "fa_common.cuh", "fa_fwd.cuh", "fa_bwd.cuh",
                                      "fa_decode.cuh", "fa_blockmask.cuh", "fa_sm100.cuh", "fa_fwd_tc.cuh", "fa_bwd_items.cuh", "fa_bwd_tc.cuh", "fa_bwd_tc128.cuh", "fa_bwd_f32.cuh", "fa_selftest.cuh"};
std::string g_templates_hash;
int templates_hash(std::string& out) {
  if (g_templates_hash.empty()) {
    std::string all;
    for (const char* f : kTemplateFiles) {
      std::string s;
      if (read_file(kernel_dir() + "/" + f, s)) all += s;
      all += "\n--\n";
    }
    if (all.size() < 200) return fail(FA_ECOMPILE, "kernel templates not found in '" + kernel_dir() + "'");
    g_templates_hash = hash_hex(all);
  }
  out = g_templates_hash;
  return FA_OK;
}

// ---- run-time compilation --------------------------------------------------------------
int nvrtc_compile(const std::string& src, const std::vector<std::string>& opts, std::string& cubin) {
  nvrtcProgram prog;
  nvrtcResult r = nvrtcCreateProgram(&prog, src.c_str(), "flaxattn_kernel.cu", 0, nullptr, nullptr);
  if (r != NVRTC_SUCCESS) return fail(FA_ECOMPILE, std::string("nvrtcCreateProgram: ") + nvrtcGetErrorString(r));
  std::vector<const char*> o;
  for (auto& s : opts) o.push_back(s.c_str());
  r = nvrtcCompileProgram(prog, (int)o.size(), o.data());
  if (r != NVRTC_SUCCESS) {
    size_t n = 0;
    nvrtcGetProgramLogSize(prog, &n);
    std::string log(n, '\0');
    if (n) nvrtcGetProgramLog(prog, &log[0]);
    nvrtcDestroyProgram(&prog);
    return fail(FA_ECOMPILE, std::string("kernel compilation failed: ") + nvrtcGetErrorString(r) + "\n" + log);
  }
  size_t n = 0;
  r = nvrtcGetCUBINSize(prog, &n);
  if (r != NVRTC_SUCCESS || n == 0) {
    nvrtcDestroyProgram(&prog);
    return fail(FA_ECOMPILE, "nvrtcGetCUBINSize failed");
  }
  cubin.resize(n);
  nvrtcGetCUBIN(prog, &cubin[0]);
  nvrtcDestroyProgram(&prog);
  g_compile_count++;
  return FA_OK;
}

struct Kernel {
  std::string cubin;
  std::string entry;
  cudaLibrary_t lib = nullptr;
  cudaKernel_t fn = nullptr;
  int smem = 0;
  std::atomic<unsigned long long> ready{0};  // devices on which the kernel is loaded and its dynamic smem limit raised
  fa_module* owner = nullptr;
  // device address of the kernel image's `fa_mod_buf` table per device (null: the image has none)
  void* buf_table[64] = {nullptr};
  unsigned long long buf_table_known = 0;
};

}  // namespace

constexpr int kMaxModBuffers = FA_MAX_MOD_BUFS;

struct fa_module {
  std::string mod_source;
  bool has_score_mod = false, linear_score_mod = false;  // (as its defines say, for the choice between variants; linear: over the keys)
  std::unordered_map<uint64_t, Kernel*> kernels;  // key: kernel_key of the variant
  const void* bufs[kMaxModBuffers] = {nullptr};  // device addresses of the captured buffers of the mods
  int nbufs = 0;
};

namespace {

const char* const kDefaultMods =
    "#define FA_HAS_SCORE_MOD 0\n#define FA_HAS_MASK_MOD 0\n"
    "__device__ __forceinline__ float fa_score_mod(float s, int, int, int, int) { return s; }\n"
    "__device__ __forceinline__ float fa_score_mod_grad(float, int, int, int, int) { return 1.0f; }\n"
    "__device__ __forceinline__ bool fa_mask_mod(int, int, int, int) { return true; }\n";

// A kernel variant of a module as a number: every launch looks its kernel up by it, and the define text
// is only put together when the variant has to be compiled or fetched from the cache on disk.
enum KernelId : int { kIdFwd, kIdFwdRerun, kIdBwdRerun, kIdFwdTc, kIdBwdDq, kIdBwdDkdv, kIdBwdTc, kIdBwdF32, kIdDecode, kIdMaskScan, kIdMaskClassify, kIdSelftest };
uint64_t kernel_key(KernelId id, std::initializer_list<std::pair<int, int>> fields) {  // (value, bits)
  uint64_t k = 0;
  for (auto& f : fields) k = (k << f.second) | (uint64_t)f.first;
  return k | (uint64_t)id << 58;
}

// Returns the compiled kernel `entry` of `tmpl` with the defines `make_defines` writes (compiling if needed).
template <class MakeDefines>
int get_kernel(fa_module* m, uint64_t key, const char* tmpl, MakeDefines make_defines, const char* entry, int smem,
               Kernel** out) {
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = m->kernels.find(key);
  if (it != m->kernels.end()) {
    *out = it->second;
    return FA_OK;
  }
  const std::string defines = make_defines();
  std::string th;
  if (int rc = templates_hash(th)) return rc;
  std::string src = defines + "\n" + m->mod_source + "\n#include \"" + std::string(tmpl) + "\"\n";
  std::vector<std::string> opts = {"--gpu-architecture=sm_100a", "-std=c++17", "-lineinfo",
                                   "-I" + kernel_dir()};
  int major = 0, minor = 0;
  nvrtcVersion(&major, &minor);
  std::string h = hash_hex(src + "|" + th + "|" + std::to_string(major) + "." + std::to_string(minor));
  std::string cubin;
  const std::string cdir = cache_dir();
  const std::string cpath = cdir + "/" + h + ".cubin";
  bool from_cache = !cdir.empty() && read_file(cpath, cubin) && cubin.size() > 64;
  if (!from_cache) {
    if (int rc = nvrtc_compile(src, opts, cubin)) return rc;
    if (!cdir.empty()) {
      mkdirs(cdir);
      const std::string tmp = cpath + ".tmp" + std::to_string((long)getpid());
      std::ofstream f(tmp, std::ios::binary);
      if (f) {
        f.write(cubin.data(), (std::streamsize)cubin.size());
        f.close();
        rename(tmp.c_str(), cpath.c_str());
      }
    }
  }
  Kernel* k = new Kernel();
  k->cubin.swap(cubin);
  k->entry = entry;
  k->smem = smem;
  k->owner = m;
  m->kernels[key] = k;
  *out = k;
  return FA_OK;
}

// Loads the kernel on first launch and raises its dynamic shared-memory limit on this device.
int ready_kernel(Kernel* k) {
  int dev = 0;
  FA_CUDA_CHECK(cudaGetDevice(&dev));
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (bit != 0 && (k->ready.load(std::memory_order_acquire) & bit)) return FA_OK;
  std::lock_guard<std::mutex> lk(g_mu);
  if (k->fn == nullptr) {
    FA_CUDA_CHECK(cudaLibraryLoadData(&k->lib, k->cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
    FA_CUDA_CHECK(cudaLibraryGetKernel(&k->fn, k->lib, k->entry.c_str()));
  }
  // (the 48 KB that need no leave include static shared memory: the table of captured buffers, which a kernel has only with such mods)
  if (k->smem > 32 * 1024)
    FA_CUDA_CHECK(cudaFuncSetAttribute((const void*)k->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k->smem));
  k->ready.fetch_or(bit, std::memory_order_release);
  return FA_OK;
}

// Mods that read captured buffers find their addresses in the `fa_mod_buf` table.  Generated mods keep it
// in shared memory, filled from the kernel parameters; a hand-written mod source may declare it
// __constant__ instead, and then the table of the kernel image is rewritten, in stream order, before
// every launch of a kernel of such a module.
int upload_buffers(Kernel* k, void* stream) {
  fa_module* m = k->owner;
  if (m == nullptr) return FA_OK;
  const void* local[kMaxModBuffers];
  int n = 0;
  void* table = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    n = m->nbufs;
    if (n == 0) return FA_OK;
    for (int i = 0; i < n; ++i) local[i] = m->bufs[i];
    int dev = 0;
    FA_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(FA_EUNSUPPORTED, "device ordinal above 63");
    if (!(k->buf_table_known >> dev & 1ull)) {
      void* dptr = nullptr;
      size_t bytes = 0;
      if (cudaLibraryGetGlobal(&dptr, &bytes, k->lib, "fa_mod_buf") != cudaSuccess) {
        cudaGetLastError();  // this kernel image does not reference the table
        dptr = nullptr;
      } else if (bytes < (size_t)n * sizeof(void*)) {
        return fail(FA_EINVAL, "fa_module_set_buffers: more buffers than the mod source declares");
      }
      k->buf_table[dev] = dptr;
      k->buf_table_known |= 1ull << dev;
    }
    table = k->buf_table[dev];
  }
  if (table != nullptr)
    FA_CUDA_CHECK(cudaMemcpyAsync(table, local, (size_t)n * sizeof(void*), cudaMemcpyHostToDevice, (cudaStream_t)stream));
  return FA_OK;
}

// ---- per-kernel device times (fa_profile_enable / fa_profile_read) -----------------------
// While profiling is on, every kernel launched by an entry point is bracketed by two CUDA events
// on the caller's stream.  The records belong to the calling thread and are reset at the start of
// each fa_fwd / fa_bwd / fa_decode call; the results of the call are the same with and without.
struct ProfRecord {
  const char* name;
  cudaEvent_t e0, e1;
};
std::atomic<int> g_profile_on{0};
thread_local std::vector<ProfRecord> t_prof;        // records of the most recent call
thread_local std::vector<cudaEvent_t> t_prof_pool;  // events of this thread, reused between calls
thread_local size_t t_prof_used = 0;
thread_local int t_prof_dev = -1;

void prof_reset() {
  if (!g_profile_on.load(std::memory_order_relaxed)) return;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  if (dev != t_prof_dev) {  // events belong to the device that was current when they were made
    for (cudaEvent_t e : t_prof_pool) cudaEventDestroy(e);
    t_prof_pool.clear();
    t_prof_dev = dev;
  }
  t_prof.clear();
  t_prof_used = 0;
}
cudaEvent_t prof_event() {
  if (t_prof_used == t_prof_pool.size()) {
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
    t_prof_pool.push_back(e);
  }
  return t_prof_pool[t_prof_used++];
}
struct ProfScope {
  cudaStream_t st;
  cudaEvent_t e1 = nullptr;
  ProfScope(const char* name, void* stream) : st((cudaStream_t)stream) {
    if (!g_profile_on.load(std::memory_order_relaxed)) return;
    cudaEvent_t e0 = prof_event();
    e1 = prof_event();
    if (e0 == nullptr || e1 == nullptr) {
      e1 = nullptr;
      return;
    }
    cudaEventRecord(e0, st);
    t_prof.push_back({name, e0, e1});
  }
  ~ProfScope() {
    if (e1 != nullptr) cudaEventRecord(e1, st);
  }
};

// Every kernel of the library begins with griddepcontrol.wait, before its first access to global memory,
// and is launched with programmatic stream serialisation: its CTAs may be scheduled as soon as those of
// the kernel in front of it on the stream have all finished or let their dependents go
// (griddepcontrol.launch_dependents), and the launch itself hides behind that kernel's tail.  The wait
// returns when the kernel in front is complete and its writes are visible.
cudaLaunchConfig_t launch_config(dim3 grid, dim3 block, int smem, void* stream, cudaLaunchAttribute* attr) {
  attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr->val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = (cudaStream_t)stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}
// cluster: CTAs along x that make a thread-block cluster (grid.x is a multiple of it)
int launch(Kernel* k, dim3 grid, dim3 block, void* params, void* stream, int cluster = 1) {
  if (int rc = ready_kernel(k)) return rc;
  if (int rc = upload_buffers(k, stream)) return rc;
  void* args[] = {params};
  ProfScope prof(k->entry.c_str(), stream);
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = launch_config(grid, block, k->smem, stream, attr);
  if (cluster > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  FA_CUDA_CHECK(cudaLaunchKernelExC(&cfg, (const void*)k->fn, args));
  return FA_OK;
}
// the same for the kernels of this file
template <class... P, class... A>
int launch_here(const char* name, void (*fn)(P...), dim3 grid, dim3 block, void* stream, A... args) {
  ProfScope prof(name, stream);
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = launch_config(grid, block, 0, stream, &attr);
  FA_CUDA_CHECK(cudaLaunchKernelEx(&cfg, fn, P(args)...));
  return FA_OK;
}

// ---- configuration ---------------------------------------------------------------------
int esize(int dtype) { return dtype == FA_F32 ? 4 : 2; }
int pitch(int cols, int es) { return cols * es + 16; }
constexpr int kMaxSmem = 227 * 1024 - 128;  // (the table of captured buffers is static shared memory)

struct FwdCfg {
  int BM, BN, warps, smem;
};
int fwd_smem(int dtype, int D, int Dv, int BM, int BN) {
  const int es = esize(dtype);
  int s = BM * pitch(D, es) + 2 * BN * pitch(D, es) + 2 * BN * pitch(Dv, es);
  if (dtype == FA_F32) s += BM * pitch(BN, 4);
  return s;
}
bool divides_or_single(int tile, int block, int nblocks) { return nblocks <= 1 || block % tile == 0; }

int pick_fwd(int dtype, int D, int Dv, int Sq, const FaTables* t, FwdCfg& c) {
  struct Cand { int BM, BN, warps; };
  std::vector<Cand> cands;
  if (dtype == FA_F32) {
    cands = {{64, 64, 4}, {64, 32, 4}, {32, 32, 2}, {16, 32, 1}, {16, 16, 1}};
  } else {
    if (D <= 64 && Sq > 64) cands.push_back({128, 64, 4});
    if (D <= 128 && Sq > 64) cands.push_back({128, 64, 8});
    cands.push_back({64, 64, 4});
    cands.push_back({64, 32, 4});
    cands.push_back({32, 32, 2});
    cands.push_back({16, 32, 1});
    cands.push_back({16, 16, 1});
  }
  for (auto& x : cands) {
    if (t && t->kv_num) {
      if (!divides_or_single(x.BM, t->QB, t->nQ) || !divides_or_single(x.BN, t->KVB, t->nKV)) continue;
    }
    const int s = fwd_smem(dtype, D, Dv, x.BM, x.BN);
    if (s > kMaxSmem) continue;
    c = {x.BM, x.BN, x.warps, s};
    return FA_OK;
  }
  return fail(FA_EUNSUPPORTED, "no forward tile configuration fits this head dim / BlockMask block size "
                               "(block sizes must be multiples of 16 unless there is a single block)");
}

struct BwdCfg {
  int tile, warps, smem_dq, smem_dkdv;
};
int pick_bwd(int dtype, int D, int Dv, const FaTables* t, BwdCfg& c) {
  const int es = esize(dtype);
  for (int warps : {4, 2, 1}) {
    const int T = 16 * warps;
    if (t && t->kv_num) {
      if (!divides_or_single(T, t->QB, t->nQ) || !divides_or_single(T, t->KVB, t->nKV)) continue;
    }
    const int pq = pitch(D, es), pv = pitch(Dv, es);
    const int f32x = dtype == FA_F32 ? T * pitch(T, 4) : 0;
    const int dq = T * pq + T * pv + 2 * T * pq + 2 * T * pv + f32x;
    const int dkdv = T * pq + T * pv + 2 * T * pq + 2 * T * pv + 2 * (2 * T * 4) + f32x;
    if (dq > kMaxSmem || dkdv > kMaxSmem) continue;
    c = {T, warps, dq, dkdv};
    return FA_OK;
  }
  return fail(FA_EUNSUPPORTED, "no backward tile configuration fits this head dim / BlockMask block size");
}

struct DecCfg {
  int BM, BN, smem, stages;
  bool tma;
};
int pick_decode(int dtype, int D, int Dv, int Sq, const FaTables* t, DecCfg& c) {
  if (dtype == FA_F32) return fail(FA_EUNSUPPORTED, "the decode kernel takes fp16 / bf16 inputs");
  if (Sq > 64) return fail(FA_EUNSUPPORTED, "the decode kernel handles at most 64 query rows");
  if (t && t->kv_num && t->nQ != 1) return fail(FA_EUNSUPPORTED, "decode needs a BlockMask with a single q block");
  const int BM = Sq <= 16 ? 16 : (Sq <= 32 ? 32 : 64);
  const int CG = 4 / (BM / 16);
  for (int BN : {128, 64, 32, 16}) {
    if (BN / CG < 16) continue;
    if (D > 64 && BN > 64) continue;
    if (t && t->kv_num && !divides_or_single(BN, t->KVB, t->nKV)) continue;
    // Two buffers of K and of V: the kernel is bound by the latency its few resident warps can hide, and
    // the smaller ring lets a third CTA share the SM (B32 H8 Skv16384 D64: 0.187 ms with two
    // stages against 0.218 ms with three at one query row, 0.224 against 0.269 at sixteen).
    const int pipe = 2 * (BN * pitch(D, 2) + BN * pitch(Dv, 2));
    const int mrg = CG * BM * (Dv + 4) * 4;
    const int smem = BM * pitch(D, 2) + (pipe > mrg ? pipe : mrg);
    if (smem > kMaxSmem) continue;
    c = {BM, BN, smem, 2, false};
    return FA_OK;
  }
  return fail(FA_EUNSUPPORTED, "no decode tile configuration fits this head dim / BlockMask block size");
}

// K and V by TMA (fa_decode.cuh): up to 16 rows, head dim 64 or 128
bool decode_by_tma(DecCfg& c, int dtype, int D, int Dv) {
  if (dtype == FA_F32 || c.BM != 16 || D != Dv || !(D == 64 || D == 128)) return false;
  const int pipe = 2 * c.stages * c.BN * D * 2, mrg = 4 * c.BM * (Dv + 4) * 4;
  c.smem = c.BM * pitch(D, 2) + std::max(pipe, mrg) + (4 * c.stages * 2 + 1) * 8 + 1024;  // fa_dec::SMEM_BYTES
  c.tma = true;
  return true;
}
// the same with three buffers of K and of V, where two CTAs of up to 16 rows still share an SM then; by cp.async only for tiles of
// more than 16 KB of K and V (us, two / three: D 16, B16 H4 Skv8191, one row 15.0 / 16.4, D 32 18.1 / 21.1; D 48 32.3 / 26.5, D 96 55.5 / 47.0, D 128
// with values of 64, 16 rows 48.7 / 40.4)
bool decode_third_buffer(DecCfg& c, int D, int Dv) {
  if (!c.tma && D + Dv <= 64) return false;
  const int smem = c.smem + (c.tma ? 2 * c.BN * D * 2 + 4 * 2 * 8 : c.BN * (pitch(D, 2) + pitch(Dv, 2)));
  if (c.BM != 16 || 2 * (smem + 1024) > 228 * 1024) return false;
  c.smem = smem;
  c.stages = 3;
  return true;
}

std::string defs(std::initializer_list<std::pair<const char*, int>> kv) {
  std::string s;
  for (auto& p : kv) s += std::string("#define ") + p.first + " " + std::to_string(p.second) + "\n";
  return s;
}

// ---- argument validation ---------------------------------------------------------------
int check_tensor(const fa_tensor& t, const char* name, int es, bool required = true) {
  if (t.ptr == nullptr) return required ? fail(FA_EINVAL, std::string(name) + ": null pointer") : FA_OK;
  if (((uintptr_t)t.ptr & 15) != 0) return fail(FA_EINVAL, std::string(name) + ": pointer must be 16-byte aligned");
  if ((t.stride_b * es) % 16 || (t.stride_h * es) % 16 || (t.stride_s * es) % 16)
    return fail(FA_EINVAL, std::string(name) + ": byte strides must be multiples of 16");
  return FA_OK;
}
FaTensor cvt(const fa_tensor& t) { return FaTensor{t.ptr, t.stride_b, t.stride_h, t.stride_s}; }

int check_common(fa_module* m, const fa_attn_params* p) {
  if (!m) return fail(FA_EINVAL, "module is null");
  if (!p) return fail(FA_EINVAL, "params is null");
  if (p->dtype < FA_F16 || p->dtype > FA_F32) return fail(FA_EINVAL, "unknown dtype");
  if (p->B <= 0 || p->Hq <= 0 || p->Hkv <= 0 || p->Sq <= 0 || p->Skv <= 0)
    return fail(FA_EINVAL, "B, Hq, Hkv, Sq, Skv must be positive");
  if (p->Hq % p->Hkv) return fail(FA_EINVAL, "Hq must be a multiple of Hkv");
  if (p->D <= 0 || p->D % 16 || p->Dv <= 0 || p->Dv % 16)
    return fail(FA_EUNSUPPORTED, "head dims must be positive multiples of 16");
  if (p->Dv > p->D) return fail(FA_EINVAL, "value head dim must not exceed the query/key head dim");
  if (p->D > 256) return fail(FA_EUNSUPPORTED, "head dim above 256 is not supported");
  if (p->B > 65535 || p->Hq > 65535) return fail(FA_EUNSUPPORTED, "B and Hq must not exceed 65535");
  const int es = esize(p->dtype);
  if (int rc = check_tensor(p->q, "q", es)) return rc;
  if (int rc = check_tensor(p->k, "k", es)) return rc;
  if (int rc = check_tensor(p->v, "v", es)) return rc;
  if (int rc = check_tensor(p->o, "o", es)) return rc;
  const fa_block_tables& t = p->tables;
  if (t.kv_num_blocks) {
    if (!t.kv_indices) return fail(FA_EINVAL, "kv_indices is null");
    if ((t.full_kv_num_blocks == nullptr) != (t.full_kv_indices == nullptr))
      return fail(FA_EINVAL, "full_kv_num_blocks and full_kv_indices must be both given or both null");
    if (t.num_q_blocks <= 0 || t.num_kv_blocks <= 0 || t.q_block_size <= 0 || t.kv_block_size <= 0)
      return fail(FA_EINVAL, "BlockMask grid and block sizes must be positive");
    if (!(t.mask_B == 1 || t.mask_B == p->B) || !(t.mask_H == 1 || t.mask_H == p->Hq))
      return fail(FA_EINVAL, "BlockMask batch/head dims must be 1 or match B/Hq");
    if ((long long)t.num_q_blocks * t.q_block_size < p->Sq || (long long)t.num_kv_blocks * t.kv_block_size < p->Skv)
      return fail(FA_EINVAL, "BlockMask does not cover the sequence lengths");
  }
  if (t.mask_bits) {
    if (!t.kv_num_blocks) return fail(FA_EINVAL, "mask_bits come with the BlockMask tables they were built beside");
    if (((uintptr_t)t.mask_bits & 15) || t.mask_bits_stride % 4 || t.mask_bits_stride * 32 < p->Skv || t.mask_bits_rows < p->Sq)
      return fail(FA_EINVAL, "mask_bits: 16-byte aligned, rows of a multiple of 4 words that cover Skv, at least Sq rows");
    if (!(t.mask_bits_B == 1 || t.mask_bits_B == p->B) || !(t.mask_bits_H == 1 || t.mask_bits_H == p->Hq))
      return fail(FA_EINVAL, "mask_bits batch/head dims must be 1 or match B/Hq");
  }
  if (t.mask_bits_t) {
    if (!t.mask_bits) return fail(FA_EINVAL, "mask_bits_t comes with mask_bits");
    if (((uintptr_t)t.mask_bits_t & 15) || t.mask_bits_t_stride % 4 || t.mask_bits_t_stride * 32 < p->Sq || t.mask_bits_t_rows < p->Skv)
      return fail(FA_EINVAL, "mask_bits_t: 16-byte aligned, rows of a multiple of 4 words that cover Sq, at least Skv rows");
  }
  return FA_OK;
}

FaTables cvt_tables(const fa_block_tables& t) {
  FaTables r;
  r.kv_num = t.kv_num_blocks; r.kv_idx = t.kv_indices;
  r.full_kv_num = t.full_kv_num_blocks; r.full_kv_idx = t.full_kv_indices;
  r.q_num = t.q_num_blocks; r.q_idx = t.q_indices;
  r.full_q_num = t.full_q_num_blocks; r.full_q_idx = t.full_q_indices;
  r.mB = t.mask_B; r.mH = t.mask_H; r.nQ = t.num_q_blocks; r.nKV = t.num_kv_blocks;
  r.QB = t.q_block_size; r.KVB = t.kv_block_size;
  r.mask_bits = t.mask_bits; r.mask_stride = t.mask_bits_stride; r.mask_rows = t.mask_bits_rows;
  r.mask_B = t.mask_bits_B; r.mask_H = t.mask_bits_H;
  r.mask_bits_t = t.mask_bits_t; r.mask_t_stride = t.mask_bits_t_stride; r.mask_t_rows = t.mask_bits_t_rows;
  r.mask_hold = t.mask_bits ? t.mask_bits_hold : nullptr;
  return r;
}

// the captured buffers of a module as they are now (fa_module_set_buffers)
void fill_buffers(fa_module* m, const void* (&out)[FA_MAX_MOD_BUFS]) {
  std::lock_guard<std::mutex> lk(g_mu);
  for (int i = 0; i < FA_MAX_MOD_BUFS; ++i) out[i] = i < m->nbufs ? m->bufs[i] : nullptr;
}

void fill_params(fa_module* m, const fa_attn_params* p, FaParams& k) {
  memset(&k, 0, sizeof k);
  fill_buffers(m, k.mod_buf);
  k.q = cvt(p->q); k.k = cvt(p->k); k.v = cvt(p->v); k.o = cvt(p->o);
  k.lse = p->lse; k.status = p->status;
  k.B = p->B; k.Hq = p->Hq; k.Hkv = p->Hkv; k.Sq = p->Sq; k.Skv = p->Skv; k.D = p->D; k.Dv = p->Dv;
  k.b_off = p->b_offset; k.h_off = p->h_offset; k.scale = p->scale;
  k.t = cvt_tables(p->tables);
}

// ---- kernels that do not depend on the mods --------------------------------------------

// The eight tables of a BlockMask from the class grid, in one launch: one warp per row of the kv tables
// and per row of the q tables (the same grid read along the other axis), each writing its partial and
// its full list.  The reference orders a row by a stable descending argsort of the 0/1 block grid
// (flaxattention/core/blockmask.py:57-64): set columns ascending, then the unset columns ascending.
// The class grid may have fewer (batch, head) entries than the tables (masks that do not read the batch
// or the head index are evaluated once): a warp works a row out once and writes it to `per` of the entries that share it.  Bound
// by the writes.  (With a warp per row of every entry the lists were worked out anew for each: 64 entries of 64 x 64 blocks
// 7.0 -> 5.4 us.)
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

struct FaTableOut {
  int *num[4], *idx[4];  // partial and full lists of the kv tables, then of the q tables (null: not wanted)
};
__global__ void __launch_bounds__(128) fa_tables_kernel(const signed char* __restrict__ cls, int B, int H, int clsB, int clsH, int nQ,
                                                        int nKV, int per, FaTableOut out) {
  grid_wait();
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  // distinct rows; entries (copies) of each, this warp's share of them: copy_lo .. copy_hi - 1
  const long long n_kv_rows = (long long)clsB * clsH * nQ, n_rows = n_kv_rows + (long long)clsB * clsH * nKV;
  if (row >= n_rows) return;
  const int copies = (clsB == 1 ? B : 1) * (clsH == 1 ? H : 1);
  const int copy_lo = (int)blockIdx.y * per, copy_hi = min(copy_lo + per, copies);
  const bool transposed = row >= n_kv_rows;
  const int rows_per_bh = transposed ? nKV : nQ, cols = transposed ? nQ : nKV;
  const long long drow = transposed ? row - n_kv_rows : row;
  const long long cbh = drow / rows_per_bh;
  const int r = (int)(drow - cbh * rows_per_bh);
  const int db = (int)(cbh / clsH), dh = (int)(cbh - (long long)db * clsH);
  // copy k is entry  first + k * apart  of the tables
  const int first = (clsB == 1 ? 0 : db) * H + (clsH == 1 ? 0 : dh), apart = clsH == 1 ? 1 : H;
  const long long row0 = ((long long)first + (long long)copy_lo * apart) * rows_per_bh + r, rows_apart = (long long)apart * rows_per_bh;
  const int n_copies = copy_hi - copy_lo;
  const signed char* g = cls + cbh * (long long)nQ * nKV + (transposed ? (long long)r : (long long)r * nKV);
  const int step = transposed ? nKV : 1;
  int total[2] = {0, 0};
  for (int c0 = 0; c0 < cols; c0 += 32) {
    const int c = c0 + lane;
    const int v = c < cols ? (int)g[(long long)c * step] : 0;
    total[0] += __popc(__ballot_sync(0xffffffffu, v == 1));
    total[1] += __popc(__ballot_sync(0xffffffffu, v == 2));
  }
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    int* num = transposed ? out.num[2 + which] : out.num[which];
    int* idx = transposed ? out.idx[2 + which] : out.idx[which];
    if (num == nullptr) continue;
    int n_set = 0;
    for (int c0 = 0; c0 < cols; c0 += 32) {
      const int c = c0 + lane;
      const bool in = c < cols;
      const bool s = in && (int)g[(long long)c * step] == which + 1;
      const unsigned bs = __ballot_sync(0xffffffffu, s);
      const int before = n_set + __popc(bs & lt);  // set columns in front of this one
      const int at = s ? before : total[which] + c - before;
      if (in) {
        int* dst = idx + row0 * cols + at;
        const long long step_out = rows_apart * cols;
#pragma unroll 4
        for (int k = 0; k < n_copies; ++k, dst += step_out) *dst = c;
      }
      n_set += __popc(bs);
    }
    for (int k = lane; k < n_copies; k += 32) num[row0 + k * rows_apart] = total[which];
  }
}


// fp32 rows of 64 values as rows of three bf16 parts, [hi | mid | lo] (192 values, contiguous), for the
// tcgen05 kernels with fp32 inputs: hi is the value rounded to bf16, mid the remainder rounded, lo the
// rest.  Up to four tensors in one launch (blockIdx.y), 8 threads per row: a thread reads 32 bytes and
// writes 16 bytes of each part.  Bound by memory: 4 bytes in and 6 out per value.
//
// Infinities, NaN and values near the end of the range have no such parts (inf - inf, 0 * inf), and sums of
// products of large ones leave it.  A byte per block says whether it saw one, |x| >= 2^30 with room
// for the products of products in the backward; the fp32 kernels launched behind then do these heads over.
//
// In front of the backward the same pass does the rest of its preparation: with q it clears dQ (the kernel adds
// to it), with dO it leaves the per-row scalars nlse2 = -lse * log2(e) (-inf for rows without mass or beyond
// Sq) and ndelta = -sum_d O * dO (0 beyond Sq), padded to whole 128-row tiles.
struct FaSplitJob {
  FaTensor src;
  uint4* dst;
  int H, S, S_rows;  // S_rows: rows gone through per (batch, head), at least S
  long long rows;
  FaTensor clear;    // cleared rows (ptr null: none)
  FaTensor o;        // with it the row scalars (ptr null: none)
  const float* lse;
  float *nlse2, *ndelta;
  float* delta;      // [B, H, S]: sum_d O * dO, for the fp32 kernels
  unsigned char* beyond;  // per block of 32 rows
};
struct FaSplitJobs {
  FaSplitJob job[4];
  int* counter;  // set to zero (or null)
};
__global__ void __launch_bounds__(256) fa_split3_kernel(const __grid_constant__ FaSplitJobs jobs) {
  grid_wait();
  grid_release();
  const FaSplitJob& j = jobs.job[blockIdx.y];
  const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
  if (t == 0 && blockIdx.y == 0 && jobs.counter != nullptr) *jobs.counter = 0;
  const long long row = t >> 3;
  const int c = (int)t & 7;
  const long long bh = row / j.S_rows;
  const int s = (int)(row - bh * j.S_rows);
  const int b = (int)(bh / j.H), h = (int)(bh - (long long)b * j.H);
  auto at = [&](const FaTensor& x) {
    return (float4*)((float*)x.ptr + (long long)b * x.sb + (long long)h * x.sh + (long long)s * x.ss) + 2 * c;
  };
  const bool valid = row < j.rows && s < j.S;  // (the same for the eight threads of a row)
  unsigned largest = 0u;
  float4 lo4 = make_float4(0.f, 0.f, 0.f, 0.f), hi4 = lo4;
  if (valid) {
    lo4 = at(j.src)[0];
    hi4 = at(j.src)[1];
    const float x[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
    unsigned part[3][4];
#pragma unroll
    for (int e = 0; e < 8; ++e) largest = max(largest, __float_as_uint(x[e]) & 0x7fffffffu);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 v = make_float2(x[2 * e], x[2 * e + 1]);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const __nv_bfloat162 r = __floats2bfloat162_rn(v.x, v.y);
        part[k][e] = *reinterpret_cast<const unsigned*>(&r);
        const float2 f = __bfloat1622float2(r);
        v.x -= f.x;
        v.y -= f.y;
      }
    }
    uint4* dst = j.dst + (bh * j.S + s) * 24 + c;
#pragma unroll
    for (int k = 0; k < 3; ++k) dst[8 * k] = make_uint4(part[k][0], part[k][1], part[k][2], part[k][3]);
    if (j.clear.ptr != nullptr) at(j.clear)[0] = at(j.clear)[1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int any = __syncthreads_or(largest >= __float_as_uint(1073741824.f) ? 1 : 0);  // 2^30; inf and NaN are above it
  if (threadIdx.x == 0 && row < j.rows) j.beyond[blockIdx.x] = any ? 1 : 0;
  if (j.o.ptr == nullptr || row >= j.rows) return;
  float acc = 0.f;
  if (valid) {
    const float4 a = at(j.o)[0], d = at(j.o)[1];
    acc = a.x * lo4.x + a.y * lo4.y + a.z * lo4.z + a.w * lo4.w + d.x * hi4.x + d.y * hi4.y + d.z * hi4.z + d.w * hi4.w;
  }
  const unsigned group = 0xffu << (threadIdx.x & 24);
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) acc += __shfl_xor_sync(group, acc, off);
  if (c == 0) {
    const float l = valid ? j.lse[bh * j.S + s] : -INFINITY;
    j.nlse2[row] = l != -INFINITY ? -(l * 1.4426950408889634f) : -INFINITY;
    j.ndelta[row] = -acc;
    if (valid) j.delta[bh * j.S + s] = acc;
  }
}

// Copies ranges of memory into a snapshot (each from a 16-byte boundary on), or compares them with one.  One CTA,
// so that the verdict needs no second pass and no word set beforehand: the ranges are a few KB (the ids of
// packed documents, 16 KB at 4096 tokens: about 2 us, most of it the launch).
struct FaRanges {
  const unsigned char* src[8];
  unsigned long long bytes[8];
  int n;
};
template <bool COMPARE>
__global__ void __launch_bounds__(1024) fa_snapshot_kernel(const __grid_constant__ FaRanges r, unsigned char* snap, int* holds) {
  grid_wait();
  grid_release();
  bool differs = false;
  for (int i = 0; i < r.n; ++i) {
    const unsigned char* a = r.src[i];
    const unsigned long long n = r.bytes[i];
    unsigned long long done = 0;
    if (((uintptr_t)a & 15) == 0) {
      done = n & ~15ull;
      for (unsigned long long k = threadIdx.x * 16ull; k < done; k += 1024 * 16) {
        const uint4 x = *(const uint4*)(a + k);
        uint4* s = (uint4*)(snap + k);
        if (COMPARE) {
          const uint4 y = *s;
          differs |= ((x.x ^ y.x) | (x.y ^ y.y) | (x.z ^ y.z) | (x.w ^ y.w)) != 0u;
        } else {
          *s = x;
        }
      }
    }
    for (unsigned long long k = done + threadIdx.x; k < n; k += 1024) {
      if (COMPARE) differs |= a[k] != snap[k];
      else snap[k] = a[k];
    }
    snap += (n + 15) & ~15ull;
  }
  if (COMPARE) {
    const int any = __syncthreads_or(differs ? 1 : 0);
    if (threadIdx.x == 0) *holds = any ? 0 : 1;
  }
}

// delta[b,h,q] = sum_d O[b,h,q,d] * dO[b,h,q,d]  (flaxattention/kernel/attention.py:338-345).
// LPR lanes cooperate on one row; each lane reads 16-byte pieces.
template <int DT, int LPR>
__global__ void fa_delta_kernel(FaTensor o, FaTensor dout, float* __restrict__ delta, int Hq, int Sq, int Dv,
                                long long n_rows) {
  grid_wait();
  grid_release();
  constexpr int ES = DT == FA_F32 ? 4 : 2;
  constexpr int EPC = 16 / ES;  // elements per 16-byte chunk
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = gt / LPR;
  const int sub = (int)(gt % LPR);
  float acc = 0.f;
  if (row < n_rows) {
    const long long bh = row / Sq;
    const int q = (int)(row - bh * Sq);
    const int b = (int)(bh / Hq), h = (int)(bh - (long long)b * Hq);
    const char* po = (const char*)o.ptr + ((long long)b * o.sb + (long long)h * o.sh + (long long)q * o.ss) * ES;
    const char* pd = (const char*)dout.ptr + ((long long)b * dout.sb + (long long)h * dout.sh + (long long)q * dout.ss) * ES;
    for (int c = sub; c * EPC < Dv; c += LPR) {
      const uint4 a = *(const uint4*)(po + c * 16);
      const uint4 d = *(const uint4*)(pd + c * 16);
      const unsigned aw[4] = {a.x, a.y, a.z, a.w}, dw[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (DT == FA_F32) {
          acc += __uint_as_float(aw[i]) * __uint_as_float(dw[i]);
        } else if (DT == FA_F16) {
          const __half2 ha = *reinterpret_cast<const __half2*>(&aw[i]);
          const __half2 hd = *reinterpret_cast<const __half2*>(&dw[i]);
          const float2 fa = __half22float2(ha), fd = __half22float2(hd);
          acc += fa.x * fd.x + fa.y * fd.y;
        } else {
          acc += __uint_as_float(aw[i] << 16) * __uint_as_float(dw[i] << 16) +
                 __uint_as_float(aw[i] & 0xffff0000u) * __uint_as_float(dw[i] & 0xffff0000u);
        }
      }
    }
  }
#pragma unroll
  for (int off = LPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (row < n_rows && sub == 0) delta[row] = acc;
}

// Per-row scalars of the tcgen05 backward, padded to whole 128-row tiles so that a q tile's
// values are one aligned 512-byte run: nlse2 = -lse * log2(e) (-inf for rows without mass or
// beyond Sq, which makes p = 0 there) and ndelta = -sum_d O * dO (0 beyond Sq).
// The same pass zeroes the dQ accumulation buffer when `dq_acc` is given (D floats per padded
// row, whatever their order inside a tile): one launch and one pass less than a separate memset.
template <int DT, int LPR>
__global__ void fa_bwd_prep_kernel(FaTensor o, FaTensor dout, const float* __restrict__ lse, float* __restrict__ nlse2,
                                   float* __restrict__ ndelta, float* __restrict__ dq_acc, int* __restrict__ work_counter,
                                   int Hq, int Sq, int sq_pad, int Dv, int D, int n_bh) {
  // grid: x over groups of R * (256 / LPR) padded rows of one (batch, head), LPR lanes per row; (y, z) over the heads.
  // A thread works on R rows, 256 / LPR apart, and has the loads of all of them in flight before it uses the first
  // (Dv <= 128: at most two 16-byte pieces of O and of dO per lane and row).
  grid_wait();
  grid_release();
  constexpr int R = 4, ROWS = 256 / LPR;
  const int bh = blockIdx.y + blockIdx.z * gridDim.y;
  const int rloc = threadIdx.x / LPR, sub = threadIdx.x % LPR;
  const int q0 = blockIdx.x * (R * ROWS) + rloc;
  if (work_counter != nullptr && blockIdx.x == 0 && threadIdx.x == 0 && bh == 0) *work_counter = 0;  // the item counter of the backward kernel
  if (bh >= n_bh) return;
  const int b = bh / Hq, h = bh - b * Hq;
  const int nc = Dv / 8;  // 16-byte pieces per row
  uint4 a[R][2], d[R][2];
  float l[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int q = q0 + r * ROWS;
    const bool valid = q < Sq;
    const char* po = (const char*)o.ptr + ((long long)b * o.sb + (long long)h * o.sh + (long long)q * o.ss) * 2;
    const char* pd = (const char*)dout.ptr + ((long long)b * dout.sb + (long long)h * dout.sh + (long long)q * dout.ss) * 2;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = sub + k * LPR;
      const bool have = valid && c < nc;
      a[r][k] = have ? *(const uint4*)(po + c * 16) : make_uint4(0u, 0u, 0u, 0u);
      d[r][k] = have ? *(const uint4*)(pd + c * 16) : make_uint4(0u, 0u, 0u, 0u);
    }
    l[r] = (valid && sub == 0) ? lse[(long long)bh * Sq + q] : 0.f;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int q = q0 + r * ROWS;
    if (q >= sq_pad) continue;  // (whole lanes groups of a row leave together)
    const long long row = (long long)bh * sq_pad + q;
    if (dq_acc != nullptr) {
      float4* z = (float4*)(dq_acc + row * D);
      for (int i = sub; i < D / 4; i += LPR) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const unsigned aw[4] = {a[r][k].x, a[r][k].y, a[r][k].z, a[r][k].w}, dw[4] = {d[r][k].x, d[r][k].y, d[r][k].z, d[r][k].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (DT == FA_F16) {
          const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&aw[i]));
          const float2 fd = __half22float2(*reinterpret_cast<const __half2*>(&dw[i]));
          acc += fa.x * fd.x + fa.y * fd.y;
        } else {
          acc += __uint_as_float(aw[i] << 16) * __uint_as_float(dw[i] << 16) +
                 __uint_as_float(aw[i] & 0xffff0000u) * __uint_as_float(dw[i] & 0xffff0000u);
        }
      }
    }
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (sub == 0) {
      const bool valid = q < Sq;
      nlse2[row] = (valid && l[r] != -INFINITY) ? -l[r] * 1.4426950408889634f : -INFINITY;
      ndelta[row] = valid ? -acc : 0.f;
    }
  }
}

// dq = scale * dq_acc for the tcgen05 backward.  The fp32 accumulation buffer holds, per (b, h, 128-row q tile), D / 32 blocks
// of [128 rows][32 columns], and the eight 16-byte chunks of a block row r sit at position k ^ (r & 7).
template <int DT, int D>
__global__ void fa_dq_convert_kernel(const float* __restrict__ acc, FaTensor dq, int Hq, int Sq, int sq_pad, float scale,
                                     int n_bh) {
  // grid: x over the rows of one (batch, head), one 8-element output chunk per thread; (y, z) over the heads
  grid_wait();
  const int bh = blockIdx.y + blockIdx.z * gridDim.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int k8 = i % (D / 8), q = i / (D / 8);
  if (bh >= n_bh || q >= Sq) return;
  const int b = bh / Hq, h = bh - b * Hq;
  const int r = q & 127, c = 2 * (k8 & 3);
  const float* src = acc + ((long long)bh * sq_pad + (q - r)) * D + (k8 >> 2) * (128 * 32) + r * 32;
  const float4 lo = *(const float4*)(src + ((c ^ (r & 7)) * 4));
  const float4 hi = *(const float4*)(src + (((c + 1) ^ (r & 7)) * 4));
  char* dst = (char*)dq.ptr + ((long long)b * dq.sb + (long long)h * dq.sh + (long long)q * dq.ss) * 2 + k8 * 16;
  if (DT == FA_F16) {
    __half2 o[4] = {__floats2half2_rn(lo.x * scale, lo.y * scale), __floats2half2_rn(lo.z * scale, lo.w * scale),
                    __floats2half2_rn(hi.x * scale, hi.y * scale), __floats2half2_rn(hi.z * scale, hi.w * scale)};
    *(uint4*)dst = *reinterpret_cast<uint4*>(o);
  } else {
    __nv_bfloat162 o[4] = {__floats2bfloat162_rn(lo.x * scale, lo.y * scale), __floats2bfloat162_rn(lo.z * scale, lo.w * scale),
                           __floats2bfloat162_rn(hi.x * scale, hi.y * scale), __floats2bfloat162_rn(hi.z * scale, hi.w * scale)};
    *(uint4*)dst = *reinterpret_cast<uint4*>(o);
  }
}

// Combines the per-split partial results of the decode kernels: one warp per output row.  Lane s takes the (max, sum)
// pair of split s and its weight 2^(m_s - m*), 32 splits at a time; the weights then go round by shuffle.  A lane owns four
// columns, and where the row has fewer than 128 the warp takes several splits at once; the reads of eight rounds
// are under way together (one at a time, the latency of each was paid in turn: half a microsecond per split), of two where
// that takes all splits: many rows of few splits are bound by instructions and by the warps that their registers let on an SM.
// WIDE: more than 128 columns.
template <int DT, int U, bool WIDE>
__global__ void fa_decode_combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                         FaTensor o, float* __restrict__ lse, int Hq, int Sq, int Dv, int ns,
                                         long long n_rows) {
  grid_wait();
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n_rows) return;
  const int lane = threadIdx.x & 31;
  const long long bh = row / Sq;
  const int q = (int)(row - bh * Sq);
  const int b = (int)(bh / Hq), h = (int)(bh - (long long)b * Hq);
  auto prow = [&](int s) -> long long { return (bh * ns + s) * Sq + q; };
  float mstar = -INFINITY;
  for (int s0 = 0; s0 < ns; s0 += 32)
    if (s0 + lane < ns) mstar = fmaxf(mstar, part_ml[prow(s0 + lane) * 2]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mstar = fmaxf(mstar, __shfl_xor_sync(0xffffffffu, mstar, off));
  const int groups = Dv >> 2;                           // of four columns
  const int per = groups < 32 ? groups : 32;            // lanes of a split
  const int sub = 32 / per, mine = lane / per;          // splits at once; this lane's (beyond sub: idle)
  const int c0 = (lane - mine * per) * 4;               // first column; head dims above 128: and 128 columns on
  const bool active = mine < sub, second = WIDE && c0 + 128 < Dv;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), acc2 = acc;
  float lstar = 0.f;
  for (int s0 = 0; s0 < ns; s0 += 32) {
    float w = 0.f;
    if (s0 + lane < ns) {
      const float2 ml = *(const float2*)(part_ml + prow(s0 + lane) * 2);
      w = ml.x == -INFINITY ? 0.f : exp2f(ml.x - mstar);
      lstar += w * ml.y;
    }
    const int cnt = ns - s0 < 32 ? ns - s0 : 32;
    for (int t0 = 0; t0 < cnt; t0 += U * sub) {
      float wt[U];
      float4 x[U], y[WIDE ? U : 1];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + u * sub + mine;
        wt[u] = __shfl_sync(0xffffffffu, w, t & 31);
        if (!active || t >= cnt) wt[u] = 0.f;
        const float* src = part_o + prow(s0 + t) * Dv + c0;
        x[u] = wt[u] != 0.f ? *(const float4*)src : make_float4(0.f, 0.f, 0.f, 0.f);
        if (WIDE) y[u] = wt[u] != 0.f && second ? *(const float4*)(src + 128) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        acc.x += wt[u] * x[u].x; acc.y += wt[u] * x[u].y; acc.z += wt[u] * x[u].z; acc.w += wt[u] * x[u].w;
        if (WIDE) { acc2.x += wt[u] * y[u].x; acc2.y += wt[u] * y[u].y; acc2.z += wt[u] * y[u].z; acc2.w += wt[u] * y[u].w; }
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) lstar += __shfl_xor_sync(0xffffffffu, lstar, off);
  const float4 own = acc;
  for (int k = 1; k < sub; ++k) {
    const int from = (lane + k * per) & 31;  // (lanes of the first split add the others' sums up)
    acc.x += __shfl_sync(0xffffffffu, own.x, from);
    acc.y += __shfl_sync(0xffffffffu, own.y, from);
    acc.z += __shfl_sync(0xffffffffu, own.z, from);
    acc.w += __shfl_sync(0xffffffffu, own.w, from);
  }
  if (lane == 0 && lse != nullptr) lse[row] = lstar > 0.f ? (mstar + log2f(lstar)) * 0.6931471805599453f : -INFINITY;
  if (mine != 0) return;
  const float inv = lstar > 0.f ? 1.f / lstar : 0.f;
  char* og = (char*)o.ptr + ((long long)b * o.sb + (long long)h * o.sh + (long long)q * o.ss + c0) * 2;
  auto put = [&](char* dst, const float4& v) {
    uint2 r;
    if (DT == FA_F16) {
      const __half2 lo = __floats2half2_rn(v.x * inv, v.y * inv), hi = __floats2half2_rn(v.z * inv, v.w * inv);
      r = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
    } else {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x * inv, v.y * inv), hi = __floats2bfloat162_rn(v.z * inv, v.w * inv);
      r = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
    }
    *(uint2*)dst = r;
  };
  put(og, acc);
  if (second) put(og + 256, acc2);
}

}  // namespace

// ======================================================================================
// C ABI
// ======================================================================================
extern "C" {

const char* fa_last_error(void) { return g_err.c_str(); }
int fa_version(void) { return 100; }

int fa_set_kernel_dir(const char* path) {
  if (!path) return fail(FA_EINVAL, "path is null");
  std::lock_guard<std::mutex> lk(g_mu);
  g_kernel_dir = path;
  g_templates_hash.clear();
  return FA_OK;
}
int fa_set_cache_dir(const char* path) {
  if (!path) return fail(FA_EINVAL, "path is null");
  std::lock_guard<std::mutex> lk(g_mu);
  g_cache_dir = path;
  g_cache_dir_set = true;
  return FA_OK;
}
int fa_compile_count(void) { return g_compile_count.load(); }

int fa_profile_enable(int on) {
  g_profile_on.store(on ? 1 : 0);
  return FA_OK;
}
int fa_profile_read(int max_kernels, float* ms, const char** names) {
  const int n = (int)t_prof.size();
  if (n == 0) return 0;
  if (max_kernels > 0 && (!ms || !names)) return fail(FA_EINVAL, "ms and names are required");
  FA_CUDA_CHECK(cudaEventSynchronize(t_prof.back().e1));
  for (int i = 0; i < n && i < max_kernels; ++i) {
    FA_CUDA_CHECK(cudaEventElapsedTime(&ms[i], t_prof[i].e0, t_prof[i].e1));
    names[i] = t_prof[i].name;
  }
  return n;
}

int fa_selftest_bounded_wait(unsigned long long limit_ns, int* status, int* gave_up, unsigned long long* waited_ns,
                             void* stream) {
  if (!status || !gave_up || !waited_ns) return fail(FA_EINVAL, "status, gave_up and waited_ns are required");
  if (limit_ns < 1000ull || limit_ns > 100000000ull) return fail(FA_EINVAL, "limit between 1 us and 100 ms");
  static fa_module* mod = nullptr;  // owns the compiled self-test kernels (one per limit)
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!mod) {
      mod = new fa_module();
      mod->mod_source = kDefaultMods;
    }
  }
  Kernel* k = nullptr;
  const auto defs = [&] { return "#define FA_WAIT_LIMIT_NS " + std::to_string(limit_ns) + "ull\n"; };
  if (int rc = get_kernel(mod, kernel_key(kIdSelftest, {{(int)limit_ns, 32}}), "fa_selftest.cuh", defs, "fa_wait_selftest_kernel", 0, &k))
    return rc;
  struct { int* status; int* gave_up; unsigned long long* waited_ns; } prm = {status, gave_up, waited_ns};
  return launch(k, dim3(1), dim3(64), &prm, stream);
}

int fa_module_create(const char* mod_source, fa_module** out) {
  if (!out) return fail(FA_EINVAL, "out is null");
  fa_module* m = new fa_module();
  m->mod_source = (mod_source && *mod_source) ? mod_source : kDefaultMods;
  m->has_score_mod = m->mod_source.find("#define FA_HAS_SCORE_MOD 1") != std::string::npos;
  m->linear_score_mod = m->mod_source.find("#define FA_SCORE_LINEAR_KV 1") != std::string::npos;
  *out = m;
  return FA_OK;
}

int fa_module_set_buffers(fa_module* m, const void* const* ptrs, int n) {
  if (!m) return fail(FA_EINVAL, "module is null");
  if (n < 0 || n > kMaxModBuffers) return fail(FA_EINVAL, "between 0 and 8 captured buffers");
  if (n > 0 && !ptrs) return fail(FA_EINVAL, "ptrs is null");
  for (int i = 0; i < n; ++i)
    if (!ptrs[i]) return fail(FA_EINVAL, "captured buffer " + std::to_string(i) + " is null");
  std::lock_guard<std::mutex> lk(g_mu);
  for (int i = 0; i < n; ++i) m->bufs[i] = ptrs[i];
  m->nbufs = n;
  return FA_OK;
}

void fa_module_destroy(fa_module* m) {
  if (!m) return;
  for (auto& kv : m->kernels) {
    if (kv.second->lib) cudaLibraryUnload(kv.second->lib);
    delete kv.second;
  }
  delete m;
}

}  // extern "C"

namespace {

int round_flag(int dtype, int flags) { return (dtype != FA_F32 && (flags & FA_FLAG_ROUND_SCORES)) ? 1 : 0; }

int get_fwd_kernel(fa_module* m, int dtype, int D, int Dv, int flags, const FwdCfg& c, Kernel** k, bool rerun = false) {
  const int rnd = round_flag(dtype, flags);
  return get_kernel(m, kernel_key(rerun ? kIdFwdRerun : kIdFwd, {{dtype, 2}, {D, 9}, {Dv, 9}, {c.BM, 9}, {c.BN, 9}, {c.warps, 5}, {rnd, 1}}), "fa_fwd.cuh",
                    [&] { return defs({{"FA_DTYPE", dtype}, {"FA_D", D}, {"FA_DV", Dv}, {"FA_BM", c.BM}, {"FA_BN", c.BN},
                                       {"FA_WARPS", c.warps}, {"FA_ROUND_SCORES", rnd}, {"FA_RERUN", rerun}}); },
                    rerun ? "fa_fwd_rerun_kernel" : "fa_fwd_kernel", c.smem, k);
}
int get_bwd_kernel(fa_module* m, int dtype, int D, int Dv, int flags, const BwdCfg& c, bool dq, Kernel** k) {
  const int rnd = round_flag(dtype, flags);
  return get_kernel(m, kernel_key(dq ? kIdBwdDq : kIdBwdDkdv, {{dtype, 2}, {D, 9}, {Dv, 9}, {c.tile, 9}, {c.warps, 5}, {rnd, 1}}),
                    "fa_bwd.cuh",
                    [&] { return defs({{"FA_DTYPE", dtype}, {"FA_D", D}, {"FA_DV", Dv}, {"FA_BQ", c.tile}, {"FA_BK", c.tile},
                                       {"FA_WARPS", c.warps}, {"FA_ROUND_SCORES", rnd}}); },
                    dq ? "fa_bwd_dq_kernel" : "fa_bwd_dkdv_kernel", dq ? c.smem_dq : c.smem_dkdv, k);
}
int get_bwd_rerun_kernel(fa_module* m, int dtype, int D, int Dv, const BwdCfg& c, Kernel** k) {
  return get_kernel(m, kernel_key(kIdBwdRerun, {{dtype, 2}, {D, 9}, {Dv, 9}, {c.tile, 9}, {c.warps, 5}}), "fa_bwd.cuh",
                    [&] { return defs({{"FA_DTYPE", dtype}, {"FA_D", D}, {"FA_DV", Dv}, {"FA_BQ", c.tile}, {"FA_BK", c.tile},
                                       {"FA_WARPS", c.warps}, {"FA_ROUND_SCORES", 0}, {"FA_RERUN", 1}}); },
                    "fa_bwd_rerun_kernel", std::max(c.smem_dq, c.smem_dkdv), k);
}
int get_decode_kernel(fa_module* m, int dtype, int D, int Dv, int flags, const DecCfg& c, bool pack, bool cluster, bool two, Kernel** k) {
  const int rnd = round_flag(dtype, flags);
  return get_kernel(m, kernel_key(kIdDecode, {{dtype, 2}, {D, 9}, {Dv, 9}, {c.BM, 9}, {c.BN, 9}, {rnd, 1}, {pack ? 1 : 0, 1}, {cluster ? 1 : 0, 1}, {two ? 1 : 0, 1}, {c.stages, 2}, {c.tma ? 1 : 0, 1}}),
                    "fa_decode.cuh",
                    [&] { return defs({{"FA_DTYPE", dtype}, {"FA_D", D}, {"FA_DV", Dv}, {"FA_BM", c.BM}, {"FA_BN", c.BN},
                                       {"FA_ROUND_SCORES", rnd}, {"FA_PACK_HEADS", pack ? 1 : 0}, {"FA_CLUSTER", cluster ? 1 : 0},
                                       {"FA_TWO_PARTS", two ? 1 : 0}, {"FA_STAGES", c.stages}, {"FA_TMA", c.tma ? 1 : 0}}); },
                    "fa_decode_kernel", c.smem, k);
}
// Grouped-query decode: the G query heads of a kv head share one CTA (their G * Sq rows form one
// tile and K / V are read once) when the rows fit a tile and the kv walk is the same for every
// head of the group, i.e. there are no tables or the tables are broadcast over the heads.
bool decode_packs_heads(const fa_attn_params* p) {
  if (p->Hkv <= 0 || p->Hq % p->Hkv) return false;
  const int G = p->Hq / p->Hkv;
  if (G <= 1 || p->dtype == FA_F32 || (long long)G * p->Sq > 64) return false;
  return p->tables.kv_num_blocks == nullptr || p->tables.mask_H == 1;
}
// ---- tcgen05 forward: TMA tensor maps and dispatch -----------------------------------------
struct alignas(64) FaTensorMapHost {
  unsigned long long v[16];
};
static_assert(sizeof(FaTensorMapHost) == sizeof(CUtensorMap), "tensor map size");
struct FaTcParamsHost {
  FaParams p;
  FaTensorMapHost tq, tk, tv, to;
};
struct FaDecodeParamsHost {
  FaParams p;
  FaTensorMapHost tk, tv;
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode_tiled = nullptr;

int encode_fn(EncodeTiledFn* out) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_encode_tiled) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    FA_CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    if (!fn || q != cudaDriverEntryPointSuccess) return fail(FA_ECUDA, "cuTensorMapEncodeTiled is not available");
    g_encode_tiled = (EncodeTiledFn)fn;
  }
  *out = g_encode_tiled;
  return FA_OK;
}

// 4-d map (D, S, H, B) over a [.., S, D]-strided tensor; box = 128 bytes x box_rows rows, 128-byte swizzle
int make_map(FaTensorMapHost* out, int dtype, const fa_tensor& t, int D, int S, int H, int B, int box_rows = 128) {
  EncodeTiledFn enc = nullptr;
  if (int rc = encode_fn(&enc)) return rc;
  const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)S, (cuuint64_t)H, (cuuint64_t)B};
  const cuuint64_t es = (cuuint64_t)esize(dtype);
  const cuuint64_t strides[3] = {(cuuint64_t)t.stride_s * es, (cuuint64_t)t.stride_h * es, (cuuint64_t)t.stride_b * es};
  const cuuint32_t box[4] = {(cuuint32_t)(128 / es), (cuuint32_t)box_rows, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUtensorMapDataType type = dtype == FA_F16    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                   : dtype == FA_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                      : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = enc((CUtensorMap*)out, type, 4,
                   t.ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(FA_ECUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return FA_OK;
}

// Shapes the tcgen05 forward kernel covers; everything else runs on the general kernel.
bool tc_fwd_eligible(const fa_attn_params* p) {
  if (p->flags & FA_FLAG_GENERAL_KERNELS) return false;
  if (p->dtype == FA_F32) return false;
  if (p->D != p->Dv || !(p->D == 64 || p->D == 128)) return false;
  if (p->Sq < 128 || p->Skv > 32768) return false;
  if (!(p->scale > 0.f)) return false;  // the kernel takes row maxima over unscaled scores
  const fa_block_tables& t = p->tables;
  if (t.kv_num_blocks) {
    if (!(t.num_q_blocks == 1 || t.q_block_size % 128 == 0)) return false;
    if (!(t.num_kv_blocks == 1 || t.kv_block_size % 128 == 0)) return false;
  }
  // byte strides above the row must stay below 2^40 (tensor-map limit); rows are 16-byte aligned already
  return true;
}

// decode = true selects the split-KV variant of the kernel (partial results); nq: query tiles of a CTA
int get_fwd_tc_kernel(fa_module* m, int dtype, int D, int flags, Kernel** k, bool decode = false, int nq = 2) {
  // must match the shared-memory map of fa_fwd_tc.cuh (fa_tc::SMEM_BYTES)
  const int atoms = dtype == FA_F32 ? 3 : D / 64, nstage = decode ? 5 : (dtype == FA_F32 ? 1 : (D == 64 ? nq + 1 : nq));
  const int smem = nq * atoms * 16384 + 2 * nstage * atoms * 16384 + (1 + 4 * nstage + 13) * 8 + 16 + (256 + 4) * 4 +
                   2 * 256 + (256 / 32) * 4 + 1024;
  const int rnd = round_flag(dtype, flags);
  return get_kernel(m, kernel_key(kIdFwdTc, {{dtype, 2}, {D, 9}, {rnd, 1}, {decode ? 1 : 0, 1}, {nq, 2}}), "fa_fwd_tc.cuh",
                    [&] { return defs({{"FA_DTYPE", dtype}, {"FA_D", D}, {"FA_ROUND_SCORES", rnd}, {"FA_TC_DECODE", decode ? 1 : 0}, {"FA_TC_NQ", nq}}); },
                    "fa_fwd_tc_kernel", smem, k);
}

// SMs of the current device (148 on a B200; asked once per device)
int device_sm_count() {
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  cached[dev].store(n, std::memory_order_relaxed);
  return n;
}

// fp32 on the tensor cores: the operands as three bf16 parts (fa_fwd_tc.cuh).
bool tc_fwd_f32_eligible(const fa_attn_params* p) {
  if (p->flags & FA_FLAG_GENERAL_KERNELS) return false;
  if (p->dtype != FA_F32 || p->D != 64 || p->Dv != 64) return false;
  if (p->Skv > 32768 || !(p->scale > 0.f)) return false;
  const fa_block_tables& t = p->tables;
  if (t.kv_num_blocks) {
    if (!(t.num_q_blocks == 1 || t.q_block_size % 128 == 0)) return false;
    if (!(t.num_kv_blocks == 1 || t.kv_block_size % 128 == 0)) return false;
  }
  return true;
}
// Up to 64 keys the forward is one tile of the general kernel, and that is faster than splitting the operands first
// (us, parts against general: B32 H16 64x64 44.6 / 29.7, B8 H16 64x64 15.4 / 10.6, B1 H1 64x64 11.6 / 10.1; from two
// tiles on B8 H16 96x96 16.3 / 27.8, B1 H1 96x96 11.6 / 18.2).
bool fwd_f32_by_parts(const fa_attn_params* p) { return p->Skv > 64 && tc_fwd_f32_eligible(p); }
// bytes of a [B, H, S, 64] tensor as three bf16 parts
size_t split3_bytes(int B, int H, int S) { return (size_t)B * H * S * 192 * 2; }
fa_tensor split3_tensor(void* ptr, int H, int S) { return fa_tensor{ptr, (int64_t)H * S * 192, (int64_t)S * 192, 192}; }
// bytes of FaParams::beyond for `rows` rows
size_t beyond_bytes(long long rows) { return (size_t)((rows + 31) / 32 + 15) / 16 * 16; }
FaSplitJob split_job(const fa_tensor& src, void* dst, int B, int H, int S, const unsigned char** beyond) {
  FaSplitJob j;
  memset(&j, 0, sizeof j);
  j.beyond = (unsigned char*)*beyond;
  j.src = cvt(src); j.dst = (uint4*)dst; j.H = H; j.S = j.S_rows = S; j.rows = (long long)B * H * S;
  return j;
}
int launch_split3(const FaSplitJobs& jobs, int n, void* stream) {
  long long rows = 0;
  for (int i = 0; i < n; ++i) rows = std::max(rows, jobs.job[i].rows);
  return launch_here("fa_split3_kernel", fa_split3_kernel, dim3((unsigned)((rows * 8 + 255) / 256), (unsigned)n), dim3(256), stream, jobs);
}
// workspace of the forward: parts of q, k, v | bytes of the blocks with values beyond them
size_t fwd_f32_workspace(const fa_attn_params* p) {
  const long long rq = (long long)p->B * p->Hq * p->Sq, rk = (long long)p->B * p->Hkv * p->Skv;
  return split3_bytes(p->B, p->Hq, p->Sq) + 2 * split3_bytes(p->B, p->Hkv, p->Skv) + beyond_bytes(rq) + 2 * beyond_bytes(rk);
}
// CTAs of an fp32 kernel launched behind the ones that work on parts: what the SMs hold, no more than tiles
dim3 rerun_grid(long long tiles, int smem) { return dim3((unsigned)std::min<long long>(tiles, (2 * (smem + 1024) <= 228 * 1024 ? 2 : 1) * device_sm_count())); }
int launch_fwd_f32_tc(fa_module* m, const fa_attn_params* p, FaParams kp, void* workspace, void* stream) {
  Kernel *k = nullptr, *kf = nullptr;
  FwdCfg c;
  if (int rc = pick_fwd(p->dtype, p->D, p->Dv, p->Sq, &kp.t, c)) return rc;
  if (int rc = get_fwd_tc_kernel(m, p->dtype, p->D, p->flags, &k)) return rc;
  if (int rc = get_fwd_kernel(m, p->dtype, p->D, p->Dv, p->flags, c, &kf, true)) return rc;
  kp.n_q_tiles = (p->Sq + c.BM - 1) / c.BM;
  char* ws = (char*)workspace;
  char* wk = ws + split3_bytes(p->B, p->Hq, p->Sq);
  char* wv = wk + split3_bytes(p->B, p->Hkv, p->Skv);
  kp.beyond[0] = (unsigned char*)(wv + split3_bytes(p->B, p->Hkv, p->Skv));
  kp.beyond[1] = kp.beyond[0] + beyond_bytes((long long)p->B * p->Hq * p->Sq);
  kp.beyond[2] = kp.beyond[1] + beyond_bytes((long long)p->B * p->Hkv * p->Skv);
  FaSplitJobs jobs;
  memset(&jobs, 0, sizeof jobs);
  jobs.job[0] = split_job(p->q, ws, p->B, p->Hq, p->Sq, &kp.beyond[0]);
  jobs.job[1] = split_job(p->k, wk, p->B, p->Hkv, p->Skv, &kp.beyond[1]);
  jobs.job[2] = split_job(p->v, wv, p->B, p->Hkv, p->Skv, &kp.beyond[2]);
  if (int rc = launch_split3(jobs, 3, stream)) return rc;
  FaTcParamsHost tp;
  tp.p = kp;
  if (int rc = make_map(&tp.tq, FA_BF16, split3_tensor(ws, p->Hq, p->Sq), 192, p->Sq, p->Hq, p->B)) return rc;
  if (int rc = make_map(&tp.tk, FA_BF16, split3_tensor(wk, p->Hkv, p->Skv), 192, p->Skv, p->Hkv, p->B)) return rc;
  if (int rc = make_map(&tp.tv, FA_BF16, split3_tensor(wv, p->Hkv, p->Skv), 192, p->Skv, p->Hkv, p->B)) return rc;
  if (int rc = make_map(&tp.to, FA_F32, p->o, p->Dv, p->Sq, p->Hq, p->B)) return rc;
  if (int rc = launch(k, dim3(p->Hq, p->B, (p->Sq + 255) / 256), dim3(384), &tp, stream)) return rc;
  return launch(kf, rerun_grid((long long)p->B * p->Hq * kp.n_q_tiles, kf->smem), dim3(c.warps * 32), &kp, stream);
}

// Shapes the split-KV variant of the tcgen05 kernel covers (`num_splits` CTAs per (batch, head), one
// partial result per CTA and row); everything else runs on the general decode kernel.
bool tc_decode_covers(const fa_attn_params* p) {
  if (p->flags & FA_FLAG_GENERAL_KERNELS) return false;
  if (p->dtype == FA_F32) return false;
  if (p->D != 64 || p->Dv != 64) return false;
  if (p->Sq < 2 || p->Sq > 64 || p->Skv < 1024 || p->Skv > 32768) return false;
  if (!(p->scale > 0.f)) return false;
  const fa_block_tables& t = p->tables;
  if (t.kv_num_blocks) {
    if (t.num_q_blocks != 1) return false;
    if (!(t.num_kv_blocks == 1 || t.kv_block_size % 128 == 0)) return false;
  }
  return true;
}
// And those it takes.  The kernel gives every query row two threads (64 kv columns of a tile each), whatever Sq is, and streams K / V
// through TMA and a five-stage ring, one CTA to an SM and at least two splits; the general kernel's time grows with the row groups of 16,
// but two or three of its CTAs share an SM, and up to 16 rows its splits are merged in a cluster.  So the tcgen05 kernel loses up to 16
// rows, and above them where many heads over short caches make it several waves of short CTAs.  Measured (us, this one / general, D 64
// fp16, inputs from memory), heads x keys:
//   rows   64 x 1024    64 x 4096    128 x 2048   128 x 4096   256 x 1536   256 x 2048   256 x 4096   512 x 1024   512 x 1536   512 x 2048
//   17     12.2 / 12.4  21.5 / 23.4  27.1 / 23.9  37.6 / 38.4  41.3 / 28.1  47.4 / 35.2  80.5 / 76.5  61.2 / 38.8  71.2 / 53.0  81.3 / 79.6
//   32     12.3 / 13.8  21.5 / 25.4  27.6 / 25.9  38.1 / 40.9  44.1 / 29.9  50.3 / 37.1  85.1 / 87.5  66.1 / 42.3  76.2 / 56.7  86.6 / 92.7
//   33     12.6 / 17.2  22.1 / 33.6  28.1 / 34.6  39.0 / 57.8  45.5 / 42.7  51.5 / 54.5  87.0 / 114   67.7 / 58.4  78.2 / 81.0  88.5 / 119
//   64     13.3 / 19.5  22.9 / 36.4  31.8 / 38.7  42.7 / 62.2  51.1 / 46.5  57.6 / 58.3  97.6 / 135   79.8 / 65.5  90.4 / 88.7  101 / 144
// (2 to 16 rows: 64 x 2048 20.6 / 18.6 with 8 rows, 256 x 8192 115 / 94 with 16, 64 x 8192 31.6 / 31.5.)
bool tc_decode_eligible(const fa_attn_params* p) {
  if (!tc_decode_covers(p) || p->Sq <= 16) return false;
  const long long heads = (long long)p->B * p->Hq, keys = heads * p->Skv;
  return p->Sq <= 32 ? heads < 128 || p->Skv > 2048 || keys > 768 << 10 : heads < 256 || p->Skv > 1536 || keys > 512 << 10;
}
int launch_decode_tc(fa_module* m, const fa_attn_params* p, const FaParams& kp, int num_splits, void* stream) {
  Kernel* k = nullptr;
  if (int rc = get_fwd_tc_kernel(m, p->dtype, p->D, p->flags, &k, true)) return rc;
  FaTcParamsHost tp;
  tp.p = kp;
  if (int rc = make_map(&tp.tq, p->dtype, p->q, p->D, p->Sq, p->Hq, p->B, 64)) return rc;  // the queries go into a tile twice
  if (int rc = make_map(&tp.tk, p->dtype, p->k, p->D, p->Skv, p->Hkv, p->B)) return rc;
  if (int rc = make_map(&tp.tv, p->dtype, p->v, p->Dv, p->Skv, p->Hkv, p->B)) return rc;
  memset(&tp.to, 0, sizeof(tp.to));  // (the decode variant writes partial results, not the output)
  return launch(k, dim3(num_splits, p->Hq, p->B), dim3(384), &tp, stream);
}

// Query tiles of a forward CTA.  With one, two CTAs share an SM: the fixed part of a CTA is hidden and the tail of
// the grid is shorter, but a step costs more (K and V are loaded per 128 rows, and with D = 128 the products of
// the two CTAs of an SM are not kept in turn).  So it is one where there are no more tiles than SMs, and at D = 64
// up to 2048 keys.  Forward alone, us, two against one:
//   at most 148 tiles  D = 64 : S1024 22.5 / 18.4, S2048 32.8 / 28.7, S8192 100 / 84, S16384 189 / 157
//                      D = 128: S1024 24.6 / 23.4, S2048 41.0 / 38.9, S8192 127 / 121, S16384 242 / 229
//   more, D = 64       dense S2048 121 / 115, S2560 107 / 100, S3072 126 / 133, S4096 109 / 118;
//                      causal S2048 78 / 76, S2560 59 / 57, S3072 77 / 76, S4096 62 / 64
//   more, D = 128      dense S2048 152 / 152, S3072 160 / 164, S4096 139 / 145; causal 98 / 94, 98 / 98, 80 / 82
// The dense lengths cross between 2560 and 3072 keys.  Under a BlockMask that leaves few steps the fixed part weighs more:
// one where the caller says that it lists up to 12 tiles of keys per query tile (D = 64; up to 16 where these are three eighths of the key tiles or
// fewer, or with rounded scores, whose steps cost more: window 1700, 14 tiles, B2 H8 S8192 107 / 105, rounded 124 / 117) or up to 10 (D = 128).
// Two against one:
//   D = 64   B4 H8 S4096 window 256 46 / 41, 1024 74 / 70, 2000 (12.7 tiles) 97.6 / 96.6, attention sink 78 / 75, 12 documents 49 / 44, causal (16.5)
//            112 / 117; B2 H8 S8192 window 256 47 / 42, 1024 85 / 75, 2000 (15.3) 111 / 113, sink 91 / 81, documents 60 / 55, causal (32.5) 193 / 207
//   D = 128  B4 H8 S4096 the same 61 / 54, 91 / 89, -, 94 / 94, 61 / 49, 135 / 149; B2 H8 S8192 66 / 58, 108 / 102, -, 114 / 107, 71 / 63, 236 / 269;
//            B4 H16 S8192 245 / 222, 406 / 417, 437 / 389, 271 / 233; causal B8 H16 S1000 (4.5) 64 / 60, B4 H8 S2560 (10.5) 67 / 67,
//            B2 H16/4 S3001 (12.5) 87 / 91
// At D = 64 also one where the tables list half of the key tiles or fewer, so that query tiles differ (causal), and there are up to three
// tiles per SM, four if they list three eighths or fewer or the scores are rounded without a score_mod: a long and a short one share an SM, where
// two neighbours in one CTA are both long.  Two against one: causal B2 H4 S4828 69 / 54, B1 H4 S8192 101 / 83, H12 S4096 (384 tiles) 59 / 53;
// B2 H8 S4096 (512) 59 / 63, B1 H8 S8192 103 / 111, but rounded 129 / 128 and with a window of 3000 92 / 84.  (Not at D = 128, causal: 63 / 62,
// 118 / 134; nor where all tiles are alike, dense B1 H4 S8192: 97 / 112.)
// At D = 64 under any tables with a score_mod: the two tiles of a CTA then fall into step, two CTAs do not.  Two against one, ALiBi:
// causal B4 H8 S4096 130 / 127, B8 H8 250 / 237, B1 H8 S16384 454 / 421, window 3000 B2 H8 S8192 164 / 156, all keys B2 H8 S8192 490 / 422,
// S2304 43 / 42; checkerboard: 123 / 120, 233 / 222, 412 / 391, -, 455 / 394, 40.4 / 39.4.  With rounded scores the same (244 / 240 causal, 512 / 452
// all keys, B2 H8 S8192), except where the mod is linear over the keys (ALiBi: causal 247 / 257, B8 H8 S4096 263 / 270, all keys 462 / 483).
int fwd_tc_query_tiles(const fa_module* m, const fa_attn_params* p) {
  const long long tiles = (long long)p->B * p->Hq * ((p->Sq + 127) / 128), kv_tiles = (p->Skv + 127) / 128;
  if (p->tables.kv_num_blocks) {
    const int listed = (p->flags >> 8) & 0xffff;
    const bool rounded = round_flag(p->dtype, p->flags);
    const bool few = 8 * listed <= 3 * kv_tiles;
    if (listed > 0 && listed <= (p->D == 64 ? (rounded || few ? 16 : 12) : 10)) return 1;
    if (p->D == 64 && m->has_score_mod && !(rounded && m->linear_score_mod)) return 1;
    const int per_sm = 2 * listed > kv_tiles + 2 ? 0 : few || (rounded && !m->has_score_mod) ? 4 : 3;
    if (p->D == 64 && listed > 0 && tiles <= (long long)per_sm * device_sm_count()) return 1;
  }
  return (p->D == 64 && p->Skv <= 2048) || tiles <= device_sm_count() ? 1 : 2;
}
int launch_fwd_tc(fa_module* m, const fa_attn_params* p, const FaParams& kp, void* stream) {
  Kernel* k = nullptr;
  const int nq = fwd_tc_query_tiles(m, p);
  if (int rc = get_fwd_tc_kernel(m, p->dtype, p->D, p->flags, &k, false, nq)) return rc;
  FaTcParamsHost tp;
  tp.p = kp;
  if (int rc = make_map(&tp.tq, p->dtype, p->q, p->D, p->Sq, p->Hq, p->B)) return rc;
  if (int rc = make_map(&tp.tk, p->dtype, p->k, p->D, p->Skv, p->Hkv, p->B)) return rc;
  if (int rc = make_map(&tp.tv, p->dtype, p->v, p->Dv, p->Skv, p->Hkv, p->B)) return rc;
  if (int rc = make_map(&tp.to, p->dtype, p->o, p->Dv, p->Sq, p->Hq, p->B)) return rc;
  // Heads vary fastest and the query tile pair slowest (the kernel walks the pairs from the last one
  // down), so that under a causal mask the CTAs with the most kv tiles are dispatched first for
  // all heads: longest-first order keeps the tail of the grid short.
  return launch(k, dim3(p->Hq, p->B, (p->Sq + 128 * nq - 1) / (128 * nq)), dim3(nq == 1 ? 256 : 384), &tp, stream);
}

// ---- tcgen05 backward ----------------------------------------------------------------------
struct FaBwdTcParamsHost {
  FaParams p;
  FaTensorMapHost tq, tk, tv, tdo, tdk, tdv;
  float* dq_acc;
  const float* nlse2;
  const float* ndelta;
  int* work_counter;
  int chunk_heads;
};

// (query head, 128-row q tile) pairs one item of the tcgen05 backward may list (fa_btc::MAXPL, fa_b128::MAXPL)
constexpr int kBwdTcMaxPairs = 1024;

bool tc_bwd_eligible(const fa_attn_params* p) {
  if (p->flags & FA_FLAG_GENERAL_KERNELS) return false;
  if (p->dtype == FA_F32) return false;
  if (p->D != p->Dv || !(p->D == 64 || p->D == 128)) return false;
  if (p->Sq < 128 || p->Skv < 128) return false;
  // a CTA lists the (query head, q tile) pairs of an item in shared memory: at most 256 q tiles
  // of 128 rows per head, and the pairs of one item must fit the list
  const int n_qtiles = (p->Sq + 127) / 128;
  if (n_qtiles > 256) return false;
  if ((long long)n_qtiles * (p->Hq / p->Hkv) > kBwdTcMaxPairs) return false;
  const fa_block_tables& t = p->tables;
  if (t.kv_num_blocks) {
    if (!(t.num_q_blocks == 1 || t.q_block_size % 128 == 0)) return false;
    if (!(t.num_kv_blocks == 1 || t.kv_block_size % 128 == 0)) return false;
  }
  return true;
}
size_t delta_bytes(const fa_attn_params* p) { return ((size_t)p->B * p->Hq * p->Sq * sizeof(float) + 255) / 256 * 256; }
size_t rows_pad_bytes(const fa_attn_params* p) {
  const size_t sq_pad = (size_t)((p->Sq + 127) / 128) * 128;
  return ((size_t)p->B * p->Hq * sq_pad * sizeof(float) + 255) / 256 * 256;
}
size_t dq_acc_bytes(const fa_attn_params* p) {
  const size_t sq_pad = (size_t)((p->Sq + 127) / 128) * 128;
  return (size_t)p->B * p->Hq * sq_pad * p->D * sizeof(float);
}

// fp32 on the tensor cores (fa_bwd_f32.cuh)
struct FaBwdF32ParamsHost {
  FaParams p;
  FaTensorMapHost tq, tk, tv, tdo;
  const float* nlse2;
  const float* ndelta;
  int* work_counter;
};
bool tc_bwd_f32_eligible(const fa_attn_params* p) {
  if (!tc_fwd_f32_eligible(p)) return false;
  const int n_qtiles = (p->Sq + 127) / 128;
  // the pair list of an item (fa_bf32::MAXPL pairs of 64 query rows)
  return n_qtiles <= 256 && (long long)2 * n_qtiles * (p->Hq / p->Hkv) <= 512;
}
// workspace: parts of q, k, v, dO | nlse2 | ndelta | item counter | delta | bytes of the blocks with values beyond the parts
size_t bwd_f32_workspace(const fa_attn_params* p) {
  const long long rq = (long long)p->B * p->Hq * p->Sq, rk = (long long)p->B * p->Hkv * p->Skv;
  return 2 * split3_bytes(p->B, p->Hq, p->Sq) + 2 * split3_bytes(p->B, p->Hkv, p->Skv) + 2 * rows_pad_bytes(p) + 256 +
         delta_bytes(p) + beyond_bytes(rq) + 2 * beyond_bytes(rk) + rows_pad_bytes(p) / 128;
}
int get_bwd_f32_kernel(fa_module* m, Kernel** k) {
  // must match the shared-memory map of fa_bwd_f32.cuh (fa_bf32::SMEM_BYTES)
  const int smem = 9 * 16384 + 9 * 8192 + 3 * 2 * 64 * 4 + 21 * 8 + 8 + 16 + 16 + 2 * 512 * 4 + 256 + 1024;
  return get_kernel(m, kernel_key(kIdBwdF32, {}), "fa_bwd_f32.cuh", [] { return std::string(); }, "fa_bwd_f32_kernel", smem, k);
}
int launch_bwd_f32_tc(fa_module* m, const fa_attn_params* p, FaParams kp, const fa_tensor& dout, void* workspace, void* stream) {
  Kernel* k = nullptr;
  if (int rc = get_bwd_f32_kernel(m, &k)) return rc;
  Kernel* kf = nullptr;
  BwdCfg c{};
  if (int rc = pick_bwd(p->dtype, p->D, p->Dv, &kp.t, c)) return rc;
  if (int rc = get_bwd_rerun_kernel(m, p->dtype, p->D, p->Dv, c, &kf)) return rc;
  const int sq_pad = (p->Sq + 127) / 128 * 128;
  char* w[4];
  w[0] = (char*)workspace;
  w[1] = w[0] + split3_bytes(p->B, p->Hq, p->Sq);
  w[2] = w[1] + split3_bytes(p->B, p->Hkv, p->Skv);
  w[3] = w[2] + split3_bytes(p->B, p->Hkv, p->Skv);
  float* nlse2 = (float*)(w[3] + split3_bytes(p->B, p->Hq, p->Sq));
  float* ndelta = (float*)((char*)nlse2 + rows_pad_bytes(p));
  int* work_counter = (int*)((char*)ndelta + rows_pad_bytes(p));
  kp.delta = (float*)((char*)work_counter + 256);
  kp.beyond[0] = (unsigned char*)kp.delta + delta_bytes(p);
  kp.beyond[1] = kp.beyond[0] + beyond_bytes((long long)p->B * p->Hq * p->Sq);
  kp.beyond[2] = kp.beyond[1] + beyond_bytes((long long)p->B * p->Hkv * p->Skv);
  kp.beyond[3] = kp.beyond[2] + beyond_bytes((long long)p->B * p->Hkv * p->Skv);
  FaBwdF32ParamsHost tp;
  tp.p = kp;
  tp.nlse2 = nlse2;
  tp.ndelta = ndelta;
  tp.work_counter = work_counter;
  FaSplitJobs jobs;
  memset(&jobs, 0, sizeof jobs);
  jobs.counter = tp.work_counter;
  jobs.job[0] = split_job(p->q, w[0], p->B, p->Hq, p->Sq, &kp.beyond[0]);
  jobs.job[0].clear = kp.dq;
  jobs.job[1] = split_job(p->k, w[1], p->B, p->Hkv, p->Skv, &kp.beyond[1]);
  jobs.job[2] = split_job(p->v, w[2], p->B, p->Hkv, p->Skv, &kp.beyond[2]);
  FaSplitJob& jd = jobs.job[3] = split_job(dout, w[3], p->B, p->Hq, p->Sq, &kp.beyond[3]);
  jd.S_rows = sq_pad; jd.rows = (long long)p->B * p->Hq * sq_pad;
  jd.o = kp.o; jd.lse = p->lse; jd.nlse2 = nlse2; jd.ndelta = ndelta; jd.delta = kp.delta;
  if (int rc = launch_split3(jobs, 4, stream)) return rc;
  if (int rc = make_map(&tp.tq, FA_BF16, split3_tensor(w[0], p->Hq, p->Sq), 192, p->Sq, p->Hq, p->B, 64)) return rc;
  if (int rc = make_map(&tp.tk, FA_BF16, split3_tensor(w[1], p->Hkv, p->Skv), 192, p->Skv, p->Hkv, p->B)) return rc;
  if (int rc = make_map(&tp.tv, FA_BF16, split3_tensor(w[2], p->Hkv, p->Skv), 192, p->Skv, p->Hkv, p->B)) return rc;
  if (int rc = make_map(&tp.tdo, FA_BF16, split3_tensor(w[3], p->Hq, p->Sq), 192, p->Sq, p->Hq, p->B, 64)) return rc;
  const long long n_items = (long long)p->Hkv * p->B * ((p->Skv + 127) / 128);
  if (int rc = launch(k, dim3((unsigned)std::min<long long>(n_items, device_sm_count())), dim3(512), &tp, stream)) return rc;
  const int n_tiles = (std::max(p->Sq, p->Skv) + c.tile - 1) / c.tile;
  return launch(kf, rerun_grid((long long)p->B * p->Hkv * n_tiles, kf->smem), dim3(c.warps * 32), &kp, stream);
}

// kv2 (head dim 64): two K / V buffers and one of dS^T instead of one and two
int get_bwd_tc_kernel(fa_module* m, int dtype, int D, int flags, bool kv2, Kernel** k) {
  const int rnd = round_flag(dtype, flags);
  const int lists = 2 * kBwdTcMaxPairs * 4 + 64 + 1024;
  if (D == 128) {
    // must match the shared-memory map of fa_bwd_tc128.cuh (fa_b128::SMEM_BYTES): thirteen blocks of 128 rows x 128 bytes
    const int smem = 13 * 16384 + 2 * 2 * 128 * 4 + 22 * 8 + 16 + 32 + lists;
    return get_kernel(m, kernel_key(kIdBwdTc, {{dtype, 2}, {D, 9}, {rnd, 1}, {1, 2}}), "fa_bwd_tc128.cuh",
                      [&] { return defs({{"FA_DTYPE", dtype}, {"FA_ROUND_SCORES", rnd}}); }, "fa_bwd_tc_kernel", smem, k);
  }
  // must match the shared-memory map of fa_bwd_tc.cuh (fa_btc::SMEM_BYTES)
  const int kvbuf = kv2 ? 2 : 1, nstage = 3, nds = kvbuf == 1 ? 2 : 1;
  const int smem = 2 * kvbuf * 16384 + 2 * nstage * 16384 + nds * 32768 + 128 * 32 * 4 + nstage * 2 * 128 * 4 +
                   (2 + 3 * nstage + 15) * 8 + 16 + 32 + lists;
  return get_kernel(m, kernel_key(kIdBwdTc, {{dtype, 2}, {D, 9}, {rnd, 1}, {kvbuf, 2}}), "fa_bwd_tc.cuh",
                    [&] { return defs({{"FA_DTYPE", dtype}, {"FA_ROUND_SCORES", rnd}, {"FA_BWD_KV2", kvbuf == 2 ? 1 : 0}}); },
                    "fa_bwd_tc_kernel", smem, k);
}

// With a BlockMask the items are short or uneven and the variant with two K / V buffers wins or ties.  Measured (us, one K / V buffer and
// two dS^T buffers / two and one, a backward pass at head dim 64): causal B2 H8 S4096 129 / 126, B1 H8 S8192 225 / 221, B1 H2 S32768
// 808 / 804, causal + checkerboard B2 H16/4 S3001 243 / 225, causal + ALiBi B8 H8 S2048 160 / 156, packed documents B4 H8 S4096 93.4 / 92.2,
// attention sink B2 H8 S8192 173 / 172, B1 H4 S32768 563 / 565.  Without one every item has all the q tiles and two dS^T buffers
// win (dense B8 H8 S2048, see fa_bwd_tc.cuh).
bool bwd_tc_kv2(const fa_attn_params* p) { return p->D == 64 && p->tables.kv_num_blocks != nullptr; }

// (batch, kv head) pairs whose items the backward works through together (item_of in fa_bwd_items.cuh; not with two K / V buffers): as
// many as keep their dQ accumulators, Q and dO in L2 (126 MB), if that leaves an item for every SM, or three where items are uneven
// (tables: the heavy items of a late chunk end up alone otherwise).  Kernel alone at head dim 128, us, all heads together / chunks of
// 96 / 48 / 24 / 12 MB: attention sink B4 H16 S8192 856 / 807 / 814 / 818 / 824, dense B4 H8 S4096 623 / 613 / 596 / 590 / 592, causal B2 H8
// S4096 179 / 181 / 222 / 223 / 234; causal + ALiBi B4 H16 S2048 205 / 220 / 223 / 248 / 242, where the rule takes 96 MB and all would be better.
int bwd_tc_chunk_heads(const fa_attn_params* p) {
  const long long heads = (long long)p->B * p->Hkv, n_kvt = (p->Skv + 127) / 128;
  const long long per_head = (long long)(p->Hq / p->Hkv) * ((p->Sq + 127) / 128 * 128) * p->D * (4 + 2 + 2);
  const bool uneven = p->tables.kv_num_blocks != nullptr;
  const long long ch = (uneven ? 96ll << 20 : 24ll << 20) / per_head;
  return (int)(ch >= heads || ch * n_kvt < (uneven ? 3 : 1) * device_sm_count() ? heads : ch);
}

// scan = false: the kernel that takes any block size
// Groups of 32 keys that a warp of fa_mask_scan_kernel takes: all four of a sub-tile, with four warps, where the mask reads captured
// tensors (a read per query serves four groups: 8.6 us against 10.5 with eight warps for 12 documents at 4096 x 4096), else two, with
// eight warps (attention sink 8192 x 8192: 10.1 us against 11.1).
int mask_scan_groups(const fa_module* m) { return m->mod_source.find("FA_NUM_MOD_BUFS") != std::string::npos ? 4 : 2; }

int get_blockmask_kernel(fa_module* m, bool scan, Kernel** k) {
  return get_kernel(m, kernel_key(scan ? kIdMaskScan : kIdMaskClassify, {}), "fa_blockmask.cuh",
                    [&] { return scan ? "#define FA_SCAN_GROUPS " + std::to_string(mask_scan_groups(m)) + "\n" : std::string(); },
                    scan ? "fa_mask_scan_kernel" : "fa_blockmask_classify_kernel", 0, k);
}

}  // namespace

extern "C" {

int fa_module_prepare(fa_module* m, int kind, int dtype, int D, int Dv, int Sq_hint, int Skv_hint) {
  if (!m) return fail(FA_EINVAL, "module is null");
  Kernel* k = nullptr;
  switch (kind) {
    case FA_KIND_FWD: {
      FwdCfg c;
      if (int rc = pick_fwd(dtype, D, Dv, Sq_hint, nullptr, c)) return rc;
      if (dtype != FA_F32 && D == Dv && (D == 64 || D == 128) && Sq_hint >= 128)
        for (int nq : {1, 2})
          if (int rc = get_fwd_tc_kernel(m, dtype, D, 0, &k, false, nq)) return rc;
      if (dtype == FA_F32 && D == 64 && Dv == 64 && Skv_hint > 64) {
        if (int rc = get_fwd_tc_kernel(m, dtype, D, 0, &k)) return rc;
        if (int rc = get_fwd_kernel(m, dtype, D, Dv, 0, c, &k, true)) return rc;
      }
      return get_fwd_kernel(m, dtype, D, Dv, 0, c, &k);
    }
    case FA_KIND_BWD: {
      BwdCfg c;
      if (int rc = pick_bwd(dtype, D, Dv, nullptr, c)) return rc;
      if (dtype != FA_F32 && D == Dv && (D == 64 || D == 128) && Sq_hint >= 128) {
        if (int rc = get_bwd_tc_kernel(m, dtype, D, 0, false, &k)) return rc;
        if (D == 64)
          if (int rc = get_bwd_tc_kernel(m, dtype, D, 0, true, &k)) return rc;
      }
      if (dtype == FA_F32 && D == 64 && Dv == 64) {
        if (int rc = get_bwd_f32_kernel(m, &k)) return rc;
        if (int rc = get_bwd_rerun_kernel(m, dtype, D, Dv, c, &k)) return rc;
      }
      if (int rc = get_bwd_kernel(m, dtype, D, Dv, 0, c, true, &k)) return rc;
      return get_bwd_kernel(m, dtype, D, Dv, 0, c, false, &k);
    }
    case FA_KIND_DECODE: {
      DecCfg c;
      if (int rc = pick_decode(dtype, D, Dv, Sq_hint, nullptr, c)) return rc;
      if (dtype != FA_F32 && D == 64 && Dv == 64 && Sq_hint > 16)
        if (int rc = get_fwd_tc_kernel(m, dtype, D, 0, &k, true)) return rc;
      const bool two = c.BM == 16 && Sq_hint > 8 && !(D == 64 && Dv == 64 && Skv_hint >= 1024 && Skv_hint <= 32768);
      // (the first kind, by cp.async, also stands in where tensors have no tensor map; then by TMA, with two buffers and with three)
      for (int kind = 0; kind < 3; ++kind) {
        if (c.BM == 16)
          if (int rc = get_decode_kernel(m, dtype, D, Dv, 0, c, false, true, two, &k)) return rc;
        if (int rc = get_decode_kernel(m, dtype, D, Dv, 0, c, false, false, two, &k)) return rc;
        if (kind == 0 && decode_by_tma(c, dtype, D, Dv)) continue;
        if (c.stages == 3 || !decode_third_buffer(c, D, Dv)) break;
      }
      return FA_OK;
    }
    case FA_KIND_BLOCKMASK:
      if (int rc = get_blockmask_kernel(m, false, &k)) return rc;
      return get_blockmask_kernel(m, true, &k);
    default:
      return fail(FA_EUNSUPPORTED, "fa_module_prepare: unknown kind");
  }
}

int fa_fwd(fa_module* m, const fa_attn_params* p, void* stream) { return fa_fwd_ws(m, p, nullptr, 0, stream); }

size_t fa_fwd_workspace_bytes(const fa_attn_params* p) {
  if (!p || p->B <= 0 || p->Hq <= 0 || p->Hkv <= 0 || p->Sq <= 0 || p->Skv <= 0 || !fwd_f32_by_parts(p)) return 0;
  return fwd_f32_workspace(p);
}

int fa_fwd_ws(fa_module* m, const fa_attn_params* p, void* workspace, size_t workspace_bytes, void* stream) {
  if (int rc = check_common(m, p)) return rc;
  if (workspace && ((uintptr_t)workspace & 15)) return fail(FA_EINVAL, "workspace must be 16-byte aligned");
  prof_reset();
  FaParams kp;
  fill_params(m, p, kp);
  if (tc_fwd_eligible(p)) return launch_fwd_tc(m, p, kp, stream);
  const size_t ws_need = fa_fwd_workspace_bytes(p);
  if (ws_need && workspace && workspace_bytes >= ws_need) return launch_fwd_f32_tc(m, p, kp, workspace, stream);
  FwdCfg c;
  if (int rc = pick_fwd(p->dtype, p->D, p->Dv, p->Sq, &kp.t, c)) return rc;
  Kernel* k = nullptr;
  if (int rc = get_fwd_kernel(m, p->dtype, p->D, p->Dv, p->flags, c, &k)) return rc;
  kp.n_q_tiles = (p->Sq + c.BM - 1) / c.BM;
  return launch(k, dim3(kp.n_q_tiles, p->Hq, p->B), dim3(c.warps * 32), &kp, stream);
}

size_t fa_bwd_workspace_bytes(const fa_attn_params* p) {
  if (!p || p->B <= 0 || p->Hq <= 0 || p->Sq <= 0) return 0;
  if (p->Hkv > 0 && p->Hq % p->Hkv == 0 && tc_bwd_f32_eligible(p)) return bwd_f32_workspace(p);
  if (p->Hkv > 0 && p->Hq % p->Hkv == 0 && tc_bwd_eligible(p)) return 2 * rows_pad_bytes(p) + dq_acc_bytes(p) + 256;
  return delta_bytes(p);
}

int fa_bwd(fa_module* m, const fa_attn_params* p, const fa_tensor* dout, const fa_tensor* dq, const fa_tensor* dk,
           const fa_tensor* dv, void* workspace, size_t workspace_bytes, void* stream) {
  if (int rc = check_common(m, p)) return rc;
  if (!dout || !dq || !dk || !dv) return fail(FA_EINVAL, "dout, dq, dk and dv descriptors are required");
  const int es = esize(p->dtype);
  if (int rc = check_tensor(*dout, "dout", es)) return rc;
  if (int rc = check_tensor(*dq, "dq", es)) return rc;
  if (int rc = check_tensor(*dk, "dk", es)) return rc;
  if (int rc = check_tensor(*dv, "dv", es)) return rc;
  if (!p->lse) return fail(FA_EINVAL, "lse (forward logsumexp) is required for the backward pass");
  if (p->tables.kv_num_blocks && !p->tables.q_num_blocks)
    return fail(FA_EINVAL, "the backward pass needs the q tables of the BlockMask");
  if (p->tables.kv_num_blocks && ((p->tables.full_q_num_blocks == nullptr) != (p->tables.full_kv_num_blocks == nullptr)))
    return fail(FA_EINVAL, "full q tables and full kv tables must be given together");
  const size_t need = fa_bwd_workspace_bytes(p);
  if (!workspace || workspace_bytes < need) return fail(FA_EWORKSPACE, "backward workspace too small");
  prof_reset();
  FaParams kp;
  fill_params(m, p, kp);
  kp.dout = cvt(*dout); kp.dq = cvt(*dq); kp.dk = cvt(*dk); kp.dv = cvt(*dv);
  kp.delta = (float*)workspace;
  if (tc_bwd_f32_eligible(p)) return launch_bwd_f32_tc(m, p, kp, *dout, workspace, stream);
  const bool use_tc = tc_bwd_eligible(p);
  BwdCfg c{};
  Kernel *kdq = nullptr, *kdkdv = nullptr, *ktc = nullptr;
  if (use_tc) {
    if (int rc = get_bwd_tc_kernel(m, p->dtype, p->D, p->flags, bwd_tc_kv2(p), &ktc)) return rc;
  } else {
    if (int rc = pick_bwd(p->dtype, p->D, p->Dv, &kp.t, c)) return rc;
    if (int rc = get_bwd_kernel(m, p->dtype, p->D, p->Dv, p->flags, c, true, &kdq)) return rc;
    if (int rc = get_bwd_kernel(m, p->dtype, p->D, p->Dv, p->flags, c, false, &kdkdv)) return rc;
  }
  if (use_tc) {
    // workspace: nlse2 | ndelta (padded rows) | dq accumulator
    float* nlse2 = (float*)workspace;
    float* ndelta = (float*)((char*)workspace + rows_pad_bytes(p));
    float* dq_acc = (float*)((char*)workspace + 2 * rows_pad_bytes(p));
    int* work_counter = (int*)((char*)workspace + 2 * rows_pad_bytes(p) + dq_acc_bytes(p));  // zeroed by the prep kernel
    const int sq_pad = (p->Sq + 127) / 128 * 128;
    const int n_bh = p->B * p->Hq;
    const int gy = n_bh < 32768 ? n_bh : 32768;
    {
      // row scalars; the same pass clears the dQ accumulator
      // 8 lanes per row, 4 rows per thread: 128 rows per block (sq_pad is a multiple of 128)
      const dim3 grid((unsigned)(sq_pad / 128), (unsigned)gy, (unsigned)((n_bh + gy - 1) / gy));
      if (int rc = launch_here("fa_bwd_prep_kernel", p->dtype == FA_F16 ? fa_bwd_prep_kernel<FA_F16, 8> : fa_bwd_prep_kernel<FA_BF16, 8>,
                               grid, dim3(256), stream, kp.o, kp.dout, p->lse, nlse2, ndelta, dq_acc, work_counter, p->Hq, p->Sq,
                               sq_pad, p->Dv, p->D, n_bh))
        return rc;
    }
    FaBwdTcParamsHost tp;
    tp.p = kp;
    tp.dq_acc = dq_acc;
    tp.nlse2 = nlse2;
    tp.ndelta = ndelta;
    tp.work_counter = work_counter;
    tp.chunk_heads = bwd_tc_chunk_heads(p);
    if (int rc = make_map(&tp.tq, p->dtype, p->q, p->D, p->Sq, p->Hq, p->B)) return rc;
    if (int rc = make_map(&tp.tk, p->dtype, p->k, p->D, p->Skv, p->Hkv, p->B)) return rc;
    if (int rc = make_map(&tp.tv, p->dtype, p->v, p->Dv, p->Skv, p->Hkv, p->B)) return rc;
    if (int rc = make_map(&tp.tdo, p->dtype, *dout, p->Dv, p->Sq, p->Hq, p->B)) return rc;
    if (int rc = make_map(&tp.tdk, p->dtype, *dk, p->D, p->Skv, p->Hkv, p->B)) return rc;
    if (int rc = make_map(&tp.tdv, p->dtype, *dv, p->Dv, p->Skv, p->Hkv, p->B)) return rc;
    // persistent: one CTA per SM (fewer when there are fewer items), items handed out through the counter
    const long long n_items = (long long)p->Hkv * p->B * ((p->Skv + 127) / 128);
    if (int rc = launch(ktc, dim3((unsigned)std::min<long long>(n_items, device_sm_count())), dim3(512), &tp, stream)) return rc;
    {
      // one 16-byte output chunk per thread: D / 8 chunks per row
      const dim3 grid((unsigned)(((long long)sq_pad * (p->D / 8) + 255) / 256), (unsigned)gy, (unsigned)((n_bh + gy - 1) / gy));
      const auto convert = p->D == 64 ? (p->dtype == FA_F16 ? fa_dq_convert_kernel<FA_F16, 64> : fa_dq_convert_kernel<FA_BF16, 64>)
                                      : (p->dtype == FA_F16 ? fa_dq_convert_kernel<FA_F16, 128> : fa_dq_convert_kernel<FA_BF16, 128>);
      if (int rc = launch_here("fa_dq_convert_kernel", convert, grid, dim3(256), stream, dq_acc, kp.dq, p->Hq, p->Sq, sq_pad, p->scale, n_bh))
        return rc;
    }
    return FA_OK;
  }
  {
    const long long n_rows = (long long)p->B * p->Hq * p->Sq;
    const int chunks = p->Dv * es / 16;
    const int lpr = chunks >= 8 ? 8 : (chunks >= 4 ? 4 : (chunks >= 2 ? 2 : 1));
    const long long threads = n_rows * lpr;
    const unsigned blocks = (unsigned)((threads + 255) / 256);
    void (*delta)(FaTensor, FaTensor, float*, int, int, int, long long) = nullptr;
#define FA_DELTA(DT, L) delta = fa_delta_kernel<DT, L>
#define FA_DELTA_DT(L)                                      \
  do {                                                      \
    if (p->dtype == FA_F16) FA_DELTA(FA_F16, L);            \
    else if (p->dtype == FA_BF16) FA_DELTA(FA_BF16, L);     \
    else FA_DELTA(FA_F32, L);                               \
  } while (0)
    if (lpr == 8) FA_DELTA_DT(8);
    else if (lpr == 4) FA_DELTA_DT(4);
    else if (lpr == 2) FA_DELTA_DT(2);
    else FA_DELTA_DT(1);
#undef FA_DELTA_DT
#undef FA_DELTA
    if (int rc = launch_here("fa_delta_kernel", delta, dim3(blocks), dim3(256), stream, kp.o, kp.dout, kp.delta, p->Hq, p->Sq, p->Dv, n_rows))
      return rc;
  }
  if (int rc = launch(kdkdv, dim3((p->Skv + c.tile - 1) / c.tile, p->Hkv, p->B), dim3(c.warps * 32), &kp, stream))
    return rc;
  return launch(kdq, dim3((p->Sq + c.tile - 1) / c.tile, p->Hq, p->B), dim3(c.warps * 32), &kp, stream);
}

// Smallest number of CTAs per (batch, head), up to cmax, whose grid fills its last wave of `slots`
// concurrent CTAs to 95 %; the best found if none does.
static int fill_waves(long long bh, int cmax, int slots) {
  int best = 1;
  double best_eff = 0.0;
  for (int c = 1; c <= cmax; ++c) {
    const double waves = (double)(bh * c) / slots;
    const double eff = waves / (double)(long long)(waves + 0.999999);
    if (eff >= 0.95) return c;
    if (eff > best_eff + 1e-9) {
      best_eff = eff;
      best = c;
    }
  }
  return best;
}

// CTAs of the general decode kernel that share an SM: by shared memory, at most four by registers
static int decode_ctas_per_sm(const DecCfg& c) { return std::min(std::max((228 * 1024) / (c.smem + 1024), 1), 4); }

// Splits of the general decode kernel for `bh` tiles of query rows over `tiles` 128-key tiles.
//   * Two CTAs per SM, all resident at once, stream as fast as more do, and every further split costs its start and its
//     merge; at least four tiles per CTA.
//   * One split, all resident at once: it leaves SMs with one CTA beside SMs with two.  Over long caches (24 tiles per CTA and more)
//     several waves that end nearly full are faster then.
//   * More tiles of rows than that: the first count whose waves end nearly full, unless one split's do (D 64, one row, us, one split /
//     so: 512 x 4096 keys 103 / 89, 512 x 8192 208 / 167, 320 x 8192 124 / 108, 640 x 4096 113 / 108, 1024 x 4096 173 / 166; 768, whose
//     one split is 0.865 full, 127 / 128 with four).
//   * More than 16 rows: the products, not the keys' way from memory, set the pace, and what counts is a last wave that is nearly
//     full (B5 H32/8 62 rows Skv1935 D128: one split 96 us, three 87; B7 H32 64 rows Skv30000 1260 / 960 with nine).
//   * Few heads: up to FA_DECODE_MAX_CLUSTER splits are merged inside a cluster, more by the combine kernel; where even a
//     cluster per head leaves SMs idle, one CTA per SM.
// Against as many CTAs as fit with the last wave 95 % full (us, before / now): B16 H32/8 Skv8191 D128 124 / 113, B4 H32
// Skv8192 D64 76.8 / 65.6, B4 H8 Skv8192 D128 54 / 41, B32 H8 Skv2048 42.0 / 38.9.
static int general_decode_splits(long long bh, int tiles, int per_sm, int sm_count, int row_groups) {
  const int cmax = std::min(std::max(tiles / 4, 1), 64);
  if (row_groups > 1) return fill_waves(bh, cmax, per_sm * sm_count);
  const int c = (int)std::min<long long>(cmax, std::max<long long>(1, std::min(per_sm, 2) * sm_count / bh));
  if (c == 1) {
    const auto waves = [&](int k) { return (double)(bh * k) / (per_sm * sm_count); };
    const auto fill = [&](int k) { return waves(k) / (double)(long long)(waves(k) + 0.999999); };  // of the last wave and those before it
    if (bh > 2LL * sm_count) {
      if (fill(1) >= 0.86) return 1;
      for (int k = 2; k <= std::min(FA_DECODE_MAX_CLUSTER, tiles / 4); ++k)
        if (fill(k) >= 0.88) return k;
      return 1;
    }
    int best = 1;
    double best_fill = 0.88;
    for (int k = 2; k <= std::min(FA_DECODE_MAX_CLUSTER, tiles / 24); ++k)
      if (waves(k) > 1.0 && fill(k) > best_fill) {
        best = k;
        best_fill = fill(k);
      }
    return best;
  }
  if (c <= FA_DECODE_MAX_CLUSTER) return c;
  return std::max(FA_DECODE_MAX_CLUSTER, (int)std::min<long long>(c, (sm_count + bh - 1) / bh));
}

// The same where K and V come by TMA.  us, with two buffers (b2) and three (b3):
//   * More than 148 tiles of rows are not split: one wave of CTAs with no merge behind it streams at 7 TB/s (16384 keys, D 64, one row: 256
//     tiles 152 with one split, 160 with five; 320: 190 / 198; 1024 keys, 512: 26 / 28), and so does a grid of several waves with the buffers
//     that fill them (decode_third).
//   * Up to 1.15 of them per SM, 4096 keys and more, would leave SMs with one CTA beside SMs with two: two splits (D 64, 160 x 8192 keys 59 -> 55).
//     With more than 8 rows, whose products weigh more, as long as all splits are resident, from 2048 keys on (160 x 2048 25 -> 23, 192 x 8192
//     83 -> 72).
//   * Up to 148: two CTAs per SM, up to FA_DECODE_MAX_CLUSTER of them merged in a cluster.  Beyond that, head dim 128 or more than 8 rows take
//     as many (D 128, 16 x 16384 keys, 16 rows: 10 splits 43, 18 34; one row 32 / 30), others one CTA per SM.
static int tma_decode_splits(long long bh, int tiles, int sm_count, int rows, int D) {
  const int cmax = std::min(std::max(tiles / 4, 1), 64);
  if (bh > sm_count) {
    const bool two = rows > 8 ? 2 * bh <= 3LL * sm_count && tiles >= 16 : 100 * bh <= 115LL * sm_count && tiles >= 32;
    return two ? 2 : 1;
  }
  const int c = (int)std::min<long long>(cmax, 2 * sm_count / bh);
  if (c <= FA_DECODE_MAX_CLUSTER || rows > 8 || D > 64) return std::max(c, 1);
  return std::max(FA_DECODE_MAX_CLUSTER, (int)std::min<long long>(c, (sm_count + bh - 1) / bh));
}
// Three buffers (and two CTAs per SM) instead of two (and three)?  us, two / three: more than 8 rows, 256 CTAs over 8192 keys 89 / 83; few tiles per
// CTA, 64 heads x 2048 keys in four splits 11.0 / 10.7; few CTAs, D 128, 192 x 16384 keys 241 / 229.  But 256 CTAs with up to 8 rows over longer
// runs 79 / 83: with more bytes in flight than it takes, memory serves them in a worse order.  Several waves: what fills the last one better
// (512 x 2048 keys 48 / 44, 640 53 / 58).
static bool decode_third(long long ctas, int tiles_per_cta, int num_splits, int sm_count, int rows) {
  if (100 * ctas <= 2 * 87LL * sm_count) return rows > 8 || tiles_per_cta <= 8 || 10 * ctas <= 13LL * sm_count;
  if (ctas <= 3LL * sm_count || num_splits > 1) return false;
  const auto fill = [&](long long places) { return (double)ctas / (double)((ctas + places - 1) / places * places); };
  return fill(2LL * sm_count) > fill(3LL * sm_count) + 0.05;
}

int fa_decode_packs_heads(const fa_attn_params* p) { return (p && decode_packs_heads(p)) ? 1 : 0; }

int fa_decode_num_splits(const fa_attn_params* p, int sm_count) {
  if (!p || p->B <= 0 || p->Hq <= 0 || p->Skv <= 0) return 1;
  if (sm_count <= 0) sm_count = 148;
  const bool pack = decode_packs_heads(p);
  const long long bh = (long long)p->B * (pack ? p->Hkv : p->Hq);
  const int tiles = (p->Skv + 127) / 128;
  // tcgen05 kernel: one CTA per SM and split, at least eight kv tiles per CTA; its partial results
  // always go through the combine kernel, so there are at least two splits
  const auto tc_splits = [&] { return std::max(2, fill_waves(bh, std::min(std::max(tiles / 8, 1), 64), sm_count)); };
  if (!pack && tc_decode_eligible(p)) return tc_splits();
  // general kernel: as many CTAs per SM as its shared memory allows (at most four by registers)
  int per_sm = 2;
  DecCfg c{16, 0, 0, 2, false};
  if (pick_decode(p->dtype, p->D, p->Dv, pack ? p->Sq * (p->Hq / p->Hkv) : p->Sq, nullptr, c) == FA_OK) {
    per_sm = decode_ctas_per_sm(c);
  }
  const int rows = pack ? p->Sq * (p->Hq / p->Hkv) : p->Sq;
  const int n = decode_by_tma(c, p->dtype, p->D, p->Dv) ? tma_decode_splits(bh, tiles, sm_count, rows, p->D)
                                                        : general_decode_splits(bh, tiles, per_sm, sm_count, c.BM / 16);
  // Callers of fa_decode_static have room for kStaticScratchBytes of partial results.  Where this count needs more, and the one
  // that fills waves (of the tcgen05 kernel where it covers the call) does not, that one is taken: many rows over many heads,
  // whose grids have CTAs enough with either.
  if (n > 1 && fa_decode_workspace_bytes(p, n) > kStaticScratchBytes) {
    const int waves = !pack && tc_decode_covers(p) ? tc_splits() : fill_waves(bh, std::min(std::max(tiles / 4, 1), 64), per_sm * sm_count);
    if (fa_decode_workspace_bytes(p, waves) <= kStaticScratchBytes) return waves;
  }
  return n;
}

size_t fa_decode_workspace_bytes(const fa_attn_params* p, int num_splits) {
  if (!p || num_splits <= 1) return 0;
  const size_t rows = (size_t)p->B * p->Hq * num_splits * p->Sq;
  return (rows * p->Dv * sizeof(float) + 255) / 256 * 256 + (rows * 2 * sizeof(float) + 255) / 256 * 256;
}

int fa_decode(fa_module* m, const fa_attn_params* p, int num_splits, void* workspace, size_t workspace_bytes,
              void* stream) {
  if (int rc = check_common(m, p)) return rc;
  if (num_splits <= 0) num_splits = fa_decode_num_splits(p, 0);
  if (num_splits > 65535) return fail(FA_EINVAL, "too many splits");
  prof_reset();
  FaParams kp;
  fill_params(m, p, kp);
  const bool pack = decode_packs_heads(p);
  const bool tc = !pack && tc_decode_eligible(p) && num_splits >= 2;
  DecCfg c;
  if (!tc)
    if (int rc = pick_decode(p->dtype, p->D, p->Dv, pack ? p->Sq * (p->Hq / p->Hkv) : p->Sq, &kp.t, c)) return rc;
  const size_t need = fa_decode_workspace_bytes(p, num_splits);
  if (need && (!workspace || workspace_bytes < need)) return fail(FA_EWORKSPACE, "decode workspace too small");
  if (need && ((uintptr_t)workspace & 15)) return fail(FA_EINVAL, "workspace must be 16-byte aligned");
  kp.num_splits = num_splits;
  // The splits of a tile of rows are merged inside a thread-block cluster where all CTAs are resident at once: no second launch and no
  // partial results in memory (us: B8 H8 Skv2048 D64 21.4 -> 16.4, B4 H8 Skv8192 D128 46 -> 41).  Where the grid takes several waves
  // a cluster has to wait for room for all its CTAs (B32 H8 Skv16384 D64, five splits: 188 -> 197), and the partial
  // results go through memory and the combine kernel.
  // (Clusters fill the SMs of a GPC in whole: at two CTAs per SM, 288 of 296 places in clusters of six take a second round, 54 -> 78 us.)
  const long long places = tc ? 0 : std::min<long long>(2, decode_ctas_per_sm(c)) * device_sm_count();
  // (More than 16 rows: the merge of that many rows costs more inside the cluster than the combine kernel does, B1 H32/8 Skv1024 D128
  // 16 rows of each head 31.2 -> 32.9, 64 rows 26.4 -> 28.9.)
  const bool cluster = !tc && c.BM == 16 && num_splits > 1 && num_splits <= FA_DECODE_MAX_CLUSTER &&
                       (long long)p->B * (pack ? p->Hkv : p->Hq) * num_splits <= (decode_ctas_per_sm(c) > 2 ? places : places * 87 / 100);
  if (need && !cluster) {
    const size_t rows = (size_t)p->B * p->Hq * num_splits * p->Sq;
    kp.part_o = (float*)workspace;
    kp.part_ml = (float*)((char*)workspace + (rows * p->Dv * sizeof(float) + 255) / 256 * 256);
  }
  if (tc) {
    // tcgen05 kernel: num_splits CTAs per (batch, head), each writing one partial result per row
    if (int rc = launch_decode_tc(m, p, kp, num_splits, stream)) return rc;
  } else {
    Kernel* k = nullptr;
    // (the second part of P as an instruction of its own: see fa_decode.cuh)
    const bool two = c.BM == 16 && (pack ? p->Sq * (p->Hq / p->Hkv) : p->Sq) > 8 && (pack || !tc_decode_covers(p));
    FaDecodeParamsHost dp;
    dp.p = kp;
    DecCfg t = c;
    const bool by_tma = decode_by_tma(t, p->dtype, p->D, p->Dv);
    if (by_tma && make_map(&dp.tk, p->dtype, p->k, p->D, p->Skv, p->Hkv, p->B, c.BN / 4) == FA_OK &&
        make_map(&dp.tv, p->dtype, p->v, p->Dv, p->Skv, p->Hkv, p->B, c.BN / 4) == FA_OK)
      c = t;
    // (cp.async: three buffers where no SM gets more than two CTAs anyway; not for strides that no tensor map takes)
    const long long ctas = (long long)p->B * (pack ? p->Hkv : p->Hq) * num_splits;
    const int tiles = (p->Skv + 127) / 128, rows = pack ? p->Sq * (p->Hq / p->Hkv) : p->Sq;
    if (c.tma ? decode_third(ctas, (tiles + num_splits - 1) / num_splits, num_splits, device_sm_count(), rows)
              : !by_tma && ctas <= (cluster ? places * 87 / 100 : 2LL * device_sm_count()))
      decode_third_buffer(c, p->D, p->Dv);
    if (int rc = get_decode_kernel(m, p->dtype, p->D, p->Dv, p->flags, c, pack, cluster, two, &k)) return rc;
    if (int rc = launch(k, dim3(num_splits, pack ? p->Hkv : p->Hq, p->B), dim3(128), &dp, stream, cluster ? num_splits : 1)) return rc;
  }
  if (num_splits > 1 && !cluster) {
    const long long n_rows = (long long)p->B * p->Hq * p->Sq;
    const unsigned blocks = (unsigned)((n_rows + 3) / 4);
    const bool few = num_splits <= 2 * (32 / std::min(p->Dv / 4, 32)), wide = p->Dv > 128;
    const auto pick = [&](auto dt) {
      constexpr int DT = decltype(dt)::value;
      return wide ? (few ? fa_decode_combine_kernel<DT, 2, true> : fa_decode_combine_kernel<DT, 8, true>)
                  : (few ? fa_decode_combine_kernel<DT, 2, false> : fa_decode_combine_kernel<DT, 8, false>);
    };
    const auto combine = p->dtype == FA_F16 ? pick(std::integral_constant<int, FA_F16>{}) : pick(std::integral_constant<int, FA_BF16>{});
    if (int rc = launch_here("fa_decode_combine_kernel", combine, dim3(blocks), dim3(128), stream, kp.part_o, kp.part_ml, kp.o, kp.lse, p->Hq, p->Sq, p->Dv, num_splits, n_rows))
      return rc;
  }
  return FA_OK;
}

size_t fa_block_mask_workspace_bytes(int B, int H, int Q_LEN, int KV_LEN, int q_block, int kv_block) {
  if (B <= 0 || H <= 0 || Q_LEN <= 0 || KV_LEN <= 0 || q_block <= 0 || kv_block <= 0) return 0;
  const long long nQ = (Q_LEN + q_block - 1) / q_block, nKV = (KV_LEN + kv_block - 1) / kv_block;
  return (size_t)((long long)B * H * nQ * nKV);
}

int64_t fa_mask_bits_row_words(int KV_LEN) { return KV_LEN <= 0 ? 0 : (int64_t)((KV_LEN + 127) / 128) * 4; }

size_t fa_snapshot_bytes(const size_t* bytes, int n) {
  size_t total = 0;
  for (int i = 0; i < n; ++i) total += (bytes[i] + 15) & ~(size_t)15;
  return total;
}
namespace {
int snapshot(const char* name, void (*fn)(FaRanges, unsigned char*, int*), const void* const* src, const size_t* bytes, int n,
             void* snap, int32_t* holds, void* stream) {
  if (n < 1 || n > 8 || !src || !bytes) return fail(FA_EINVAL, "between 1 and 8 ranges");
  if (!snap || ((uintptr_t)snap & 15)) return fail(FA_EINVAL, "the snapshot must be 16-byte aligned");
  FaRanges r;
  memset(&r, 0, sizeof r);
  r.n = n;
  for (int i = 0; i < n; ++i) {
    if (!src[i]) return fail(FA_EINVAL, "a range is null");
    r.src[i] = (const unsigned char*)src[i];
    r.bytes[i] = bytes[i];
  }
  return launch_here(name, fn, dim3(1), dim3(1024), stream, r, (unsigned char*)snap, (int*)holds);
}
}  // namespace
int fa_snapshot(const void* const* src, const size_t* bytes, int n, void* snap, void* stream) {
  return snapshot("fa_snapshot_kernel", fa_snapshot_kernel<false>, src, bytes, n, snap, nullptr, stream);
}
int fa_snapshot_holds(const void* const* src, const size_t* bytes, int n, const void* snap, int32_t* holds, void* stream) {
  if (!holds) return fail(FA_EINVAL, "holds is null");
  return snapshot("fa_snapshot_kernel", fa_snapshot_kernel<true>, src, bytes, n, (void*)snap, holds, stream);
}

int fa_mask_bits(fa_module* m, int B, int H, int Q_LEN, int KV_LEN, int b_offset, int h_offset, uint32_t* bits,
                 void* stream) {
  if (B <= 0 || H <= 0 || Q_LEN <= 0 || KV_LEN <= 0) return fail(FA_EINVAL, "B, H, Q_LEN and KV_LEN must be positive");
  if (!bits) return fail(FA_EINVAL, "bits is null");
  fa_mask_build mb{};
  mb.B = mb.distinct_B = B; mb.H = mb.distinct_H = H;
  mb.Q_LEN = Q_LEN; mb.KV_LEN = KV_LEN; mb.q_block = 128; mb.kv_block = 128;
  mb.b_offset = b_offset; mb.h_offset = h_offset;
  mb.bits = bits;
  return fa_block_mask_build(m, &mb, stream);
}

int fa_block_mask(fa_module* m, int B, int H, int Q_LEN, int KV_LEN, int q_block, int kv_block, int b_offset,
                  int h_offset, int32_t* kv_num_blocks, int32_t* kv_indices, int32_t* full_kv_num_blocks,
                  int32_t* full_kv_indices, int32_t* q_num_blocks, int32_t* q_indices, int32_t* full_q_num_blocks,
                  int32_t* full_q_indices, void* workspace, size_t workspace_bytes, void* stream) {
  if (!kv_num_blocks || !kv_indices) return fail(FA_EINVAL, "kv_num_blocks / kv_indices are null");
  fa_mask_build mb{};
  mb.B = mb.distinct_B = B; mb.H = mb.distinct_H = H;
  mb.Q_LEN = Q_LEN; mb.KV_LEN = KV_LEN; mb.q_block = q_block; mb.kv_block = kv_block;
  mb.b_offset = b_offset; mb.h_offset = h_offset;
  mb.kv_num_blocks = kv_num_blocks; mb.kv_indices = kv_indices;
  mb.full_kv_num_blocks = full_kv_num_blocks; mb.full_kv_indices = full_kv_indices;
  mb.q_num_blocks = q_num_blocks; mb.q_indices = q_indices;
  mb.full_q_num_blocks = full_q_num_blocks; mb.full_q_indices = full_q_indices;
  mb.workspace = workspace; mb.workspace_bytes = workspace_bytes;
  return fa_block_mask_build(m, &mb, stream);
}

int fa_block_mask_build(fa_module* m, const fa_mask_build* mb, void* stream) {
  if (!m) return fail(FA_EINVAL, "module is null");
  if (!mb) return fail(FA_EINVAL, "the description is null");
  const int QB = mb->q_block, KVB = mb->kv_block;
  if (mb->B <= 0 || mb->H <= 0 || mb->Q_LEN <= 0 || mb->KV_LEN <= 0 || QB <= 0 || KVB <= 0)
    return fail(FA_EINVAL, "B, H, Q_LEN, KV_LEN and block sizes must be positive");
  if (!(mb->distinct_B == 1 || mb->distinct_B == mb->B) || !(mb->distinct_H == 1 || mb->distinct_H == mb->H))
    return fail(FA_EINVAL, "the distinct entries along batch / heads must be 1 or B / H");
  const bool tables = mb->kv_num_blocks != nullptr;
  const size_t need = fa_block_mask_workspace_bytes(mb->distinct_B, mb->distinct_H, mb->Q_LEN, mb->KV_LEN, QB, KVB);
  if (tables) {
    if (!mb->kv_indices) return fail(FA_EINVAL, "kv_num_blocks / kv_indices are null");
    if ((mb->full_kv_num_blocks == nullptr) != (mb->full_kv_indices == nullptr))
      return fail(FA_EINVAL, "full_kv_num_blocks and full_kv_indices must be both given or both null");
    if ((mb->q_num_blocks == nullptr) != (mb->q_indices == nullptr) || (mb->full_q_num_blocks == nullptr) != (mb->full_q_indices == nullptr))
      return fail(FA_EINVAL, "q tables must be given as (num, indices) pairs");
    if (mb->full_q_num_blocks && !mb->full_kv_num_blocks) return fail(FA_EINVAL, "full q tables need full kv tables");
    if (!mb->workspace || mb->workspace_bytes < need) return fail(FA_EWORKSPACE, "block-mask workspace too small");
    // Without separate full tables every non-empty block is listed as partial.
    if (!mb->full_kv_num_blocks) return fail(FA_EUNSUPPORTED, "tables without separate full blocks are not implemented");
  }
  if (((uintptr_t)mb->bits & 15) || ((uintptr_t)mb->bits_t & 15)) return fail(FA_EINVAL, "bits must be 16-byte aligned");
  const int nQ = (mb->Q_LEN + QB - 1) / QB, nKV = (mb->KV_LEN + KVB - 1) / KVB;
  const long long nbh = (long long)mb->distinct_B * mb->distinct_H;
  if ((long long)mb->B * mb->H > 65535 || nQ > 65535)
    return fail(FA_EUNSUPPORTED, "B*H and the q-block count must not exceed 65535");
  const bool words = (nQ == 1 || QB % 32 == 0) && (nKV == 1 || KVB % 32 == 0) && (long long)QB * KVB < (1ll << 31);
  if (!words && (mb->bits || mb->bits_t)) return fail(FA_EUNSUPPORTED, "bit matrices need blocks of whole 32-bit words");
  Kernel* k = nullptr;
  if (int rc = get_blockmask_kernel(m, words, &k)) return rc;
  prof_reset();
  FaMaskParams mp;
  memset(&mp, 0, sizeof mp);
  mp.cls = tables ? (signed char*)mb->workspace : nullptr;
  mp.bits = mb->bits; mp.bits_t = mb->bits_t;
  mp.stride = fa_mask_bits_row_words(mb->KV_LEN); mp.stride_t = fa_mask_bits_row_words(mb->Q_LEN);
  mp.B = mb->distinct_B; mp.H = mb->distinct_H; mp.nQ = nQ; mp.nKV = nKV; mp.QB = QB; mp.KVB = KVB;
  mp.Q_LEN = mb->Q_LEN; mp.KV_LEN = mb->KV_LEN;
  mp.b_off = mb->b_offset; mp.h_off = mb->h_offset;
  fill_buffers(m, mp.mod_buf);
  const int threads = words ? 512 / mask_scan_groups(m) : 256;
  if (int rc = launch(k, dim3(nKV, nQ, (unsigned)nbh), dim3(threads), &mp, stream)) return rc;
  if (!tables) return FA_OK;
  FaTableOut out = {{mb->kv_num_blocks, mb->full_kv_num_blocks, mb->q_num_blocks, mb->full_q_num_blocks},
                    {mb->kv_indices, mb->full_kv_indices, mb->q_indices, mb->full_q_indices}};
  const long long n_rows = nbh * ((long long)nQ + (mb->q_num_blocks || mb->full_q_num_blocks ? nKV : 0));
  // entries per warp: several, while that leaves sixteen warps per SM
  const long long copies = (long long)mb->B * mb->H / nbh;
  const int per = (int)std::min<long long>(copies, std::max<long long>(1, n_rows * copies / (16LL * device_sm_count())));
  return launch_here("fa_tables_kernel", fa_tables_kernel, dim3((unsigned)((n_rows + 3) / 4), (unsigned)((copies + per - 1) / per)), dim3(128),
                     stream, mp.cls, mb->B, mb->H, mb->distinct_B, mb->distinct_H, nQ, nKV, per, out);
}

}  // extern "C"

// ======================================================================================
// Decode without any allocation by the caller or the library
// ======================================================================================
namespace {

// Scratch for the split-KV partial results of fa_decode_static.  It is part of the loaded
// library image: every GPU that loads the library holds these bytes until the process exits.
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

std::mutex g_static_mu;
void* g_static_ptr[64] = {nullptr};

// In host code `g_static_scratch` is only a handle for the symbol, not a device address; the
// address a kernel can use has to be asked for, once per device, with that device current.
int static_scratch(void** out, void* stream) {
  int dev = 0;
  FA_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(FA_EUNSUPPORTED, "device ordinal above 63");
  // the scratch address is the current device's: a stream of another device would run the kernels there
  if (stream != nullptr && stream != (void*)cudaStreamLegacy && stream != (void*)cudaStreamPerThread) {
    int sdev = dev;
    if (cudaStreamGetDevice((cudaStream_t)stream, &sdev) == cudaSuccess && sdev != dev)
      return fail(FA_EINVAL, "fa_decode_static: the stream belongs to device " + std::to_string(sdev) +
                                 ", the current device is " + std::to_string(dev));
    cudaGetLastError();
  }
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (g_static_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    FA_CUDA_CHECK(cudaGetSymbolAddress(&ptr, g_static_scratch));
    if (ptr == nullptr) return fail(FA_ECUDA, "cudaGetSymbolAddress returned a null address");
    g_static_ptr[dev] = ptr;
  }
  *out = g_static_ptr[dev];
  return FA_OK;
}

}  // namespace

extern "C" {

size_t fa_decode_static_capacity(void) { return kStaticScratchBytes; }

int fa_decode_static(fa_module* m, const fa_attn_params* p, int num_splits, void* stream) {
  // arguments first: the sizes below are products of fields that have to be positive
  if (int rc = check_common(m, p)) return rc;
  if (p->dtype == FA_F32) return fail(FA_EUNSUPPORTED, "the decode kernel takes fp16 / bf16 inputs");
  if (p->Sq > 64) return fail(FA_EUNSUPPORTED, "the decode kernel handles at most 64 query rows");
  if (num_splits <= 0) num_splits = fa_decode_num_splits(p, 0);
  const size_t need = fa_decode_workspace_bytes(p, num_splits);
  if (need == 0) return fa_decode(m, p, num_splits, nullptr, 0, stream);  // a single split needs no scratch
  if (need > kStaticScratchBytes)
    return fail(FA_EWORKSPACE, "fa_decode_static: this problem needs " + std::to_string(need) +
                                   " bytes of split-KV scratch, the built-in scratch holds " +
                                   std::to_string(kStaticScratchBytes) + "; use fewer splits or fa_decode");
  void* ws = nullptr;
  if (int rc = static_scratch(&ws, stream)) return rc;
  return fa_decode(m, p, num_splits, ws, kStaticScratchBytes, stream);
}

}  // extern "C"
