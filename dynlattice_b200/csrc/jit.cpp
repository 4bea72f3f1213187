// NVRTC compilation of the step kernels (see jit.hpp).
#include "jit.hpp"

#include <cuda_runtime.h>
#include <nvrtc.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <map>
#include <memory>
#include <mutex>
#include <sstream>
#include <sys/stat.h>
#include <thread>
#include <vector>

#include "jit_sources.inc"  // kJitHeaderNames / kJitHeaders (generated from the .cuh files)

namespace dl {

namespace {

struct Entry {
  std::vector<cudaLibrary_t> libs;
  KernelSet ks;
};

std::mutex g_mu;
std::map<std::string, std::unique_ptr<Entry>> g_cache;

uint64_t fnv1a(const std::string &s) {
  uint64_t h = 1469598103934665603ULL;
  for (unsigned char c : s) {
    h ^= c;
    h *= 1099511628211ULL;
  }
  return h;
}

std::string cache_dir() {
  const char *d = std::getenv("DL_JIT_CACHE");
  if (d && *d) return d;
  const char *home = std::getenv("HOME");
  return std::string(home ? home : "/tmp") + "/.cache/dynlattice_b200";
}

void mkdirs(const std::string &p) {
  std::string cur;
  std::stringstream ss(p);
  std::string part;
  if (!p.empty() && p[0] == '/') cur = "/";
  while (std::getline(ss, part, '/')) {
    if (part.empty()) continue;
    cur += part + "/";
    mkdir(cur.c_str(), 0755);
  }
}

bool read_file(const std::string &path, std::vector<char> &out) {
  std::ifstream f(path, std::ios::binary);
  if (!f) return false;
  out.assign(std::istreambuf_iterator<char>(f), std::istreambuf_iterator<char>());
  return !out.empty();
}

}  // namespace

namespace {

// compile one kernel (a name expression) of `src`, which includes the embedded
// headers, for sm_100a; results cached on disk by content hash
bool compile_kernel(const std::string &src, const std::string &name, bool fp32, const std::string &tag,
                    JitKernel *out, std::string *log) {
  const char *T = fp32 ? "float" : "double";
  // the FP32 variant uses approximate (not correctly rounded) division and
  // square root; transcendentals stay accurate (small rotation angles need a
  // relative error bound).  Its error budget against the FP64 path is 1e-5.
  const char *opts32[] = {"-arch=sm_100a", "-std=c++17", "-DNDEBUG", "-prec-div=false", "-prec-sqrt=false",
                          "-ftz=true"};
  const char *opts64[] = {"-arch=sm_100a", "-std=c++17", "-DNDEBUG"};
  const char *const *opts = fp32 ? opts32 : opts64;
  const int nopts = fp32 ? 6 : 3;
  int nv_major = 0, nv_minor = 0;
  nvrtcVersion(&nv_major, &nv_minor);
  std::string full = src + (fp32 ? "|approx-div-sqrt" : "");
  full += "|" + name;
  for (size_t i = 0; i < sizeof(kJitHeaders) / sizeof(kJitHeaders[0]); ++i) full += kJitHeaders[i];
  char hbuf[64];
  std::snprintf(hbuf, sizeof hbuf, "%016llx_%d_%d_%s", static_cast<unsigned long long>(fnv1a(full)), nv_major,
                nv_minor, T);
  const std::string dir = cache_dir();
  const std::string cubin_path = dir + "/" + tag + "_" + hbuf + ".cubin";
  const std::string names_path = dir + "/" + tag + "_" + hbuf + ".names";
  {
    std::vector<char> nb;
    if (read_file(cubin_path, out->cubin) && read_file(names_path, nb)) {
      std::stringstream ns(std::string(nb.begin(), nb.end()));
      std::getline(ns, out->lowered);
      if (!out->lowered.empty()) return true;
    }
  }
  nvrtcProgram prog;
  const int nh = static_cast<int>(sizeof(kJitHeaders) / sizeof(kJitHeaders[0]));
  if (nvrtcCreateProgram(&prog, src.c_str(), "dl_jit.cu", nh, kJitHeaders, kJitHeaderNames) != NVRTC_SUCCESS) {
    if (log) *log = "nvrtcCreateProgram failed";
    return false;
  }
  nvrtcAddNameExpression(prog, name.c_str());
  nvrtcResult rc = nvrtcCompileProgram(prog, nopts, opts);
  if (rc != NVRTC_SUCCESS) {
    size_t ls = 0;
    nvrtcGetProgramLogSize(prog, &ls);
    std::string l(ls, '\0');
    nvrtcGetProgramLog(prog, &l[0]);
    if (log) *log = std::string("NVRTC: ") + nvrtcGetErrorString(rc) + "\n" + l;
    nvrtcDestroyProgram(&prog);
    return false;
  }
  size_t cs = 0;
  nvrtcGetCUBINSize(prog, &cs);
  out->cubin.resize(cs);
  nvrtcGetCUBIN(prog, out->cubin.data());
  const char *ln = nullptr;
  nvrtcGetLoweredName(prog, name.c_str(), &ln);
  out->lowered = ln ? ln : "";
  nvrtcDestroyProgram(&prog);
  // best-effort disk cache (atomic rename)
  mkdirs(dir);
  {
    std::ofstream fc(cubin_path + ".tmp", std::ios::binary);
    fc.write(out->cubin.data(), static_cast<std::streamsize>(out->cubin.size()));
  }
  {
    std::ofstream fn(names_path + ".tmp");
    fn << out->lowered << "\n";
  }
  std::rename((cubin_path + ".tmp").c_str(), cubin_path.c_str());
  std::rename((names_path + ".tmp").c_str(), names_path.c_str());
  return true;
}

// Each kernel is a program of its own, and the programs are compiled at the same
// time: twelve step kernels take 30 s one after another and 7 s on eight cores.
bool compile_kernels(const std::string &src, const std::vector<std::string> &names, bool fp32,
                     const std::string &tag, std::vector<JitKernel> *out, std::string *log) {
  const size_t n = names.size();
  out->assign(n, JitKernel{});
  std::vector<std::string> logs(n);
  std::vector<char> ok(n, 0);
  std::atomic<size_t> next{0};
  auto work = [&] {
    for (size_t i; (i = next.fetch_add(1)) < n;) {
      try {
        ok[i] = compile_kernel(src, names[i], fp32, tag, &(*out)[i], &logs[i]);
      } catch (...) {  // out of memory: not ok
      }
    }
  };
  std::vector<std::thread> helpers;
  helpers.reserve(n);
  const size_t cores = std::max(1u, std::thread::hardware_concurrency());
  try {
    while (helpers.size() + 1 < std::min(n, cores)) helpers.emplace_back(work);
  } catch (const std::exception &) {  // no more threads: those there are do the work
  }
  work();
  for (std::thread &t : helpers) t.join();
  for (size_t i = 0; i < n; ++i) {
    if (ok[i]) continue;
    if (log) *log = logs[i].empty() ? "runtime compilation ran out of memory" : logs[i];
    return false;
  }
  return true;
}

// Loads compiled kernels; false (with a message) when one cannot be.
bool load_kernels(const std::vector<JitKernel> &jk, std::vector<cudaLibrary_t> *libs, std::vector<const void *> *k,
                  std::string *log) {
  for (const JitKernel &j : jk) {
    cudaLibrary_t lib = nullptr;
    cudaKernel_t kernel = nullptr;
    if (cudaLibraryLoadData(&lib, j.cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0) != cudaSuccess) {
      cudaGetLastError();
      if (log) *log = "cudaLibraryLoadData failed";
      return false;
    }
    libs->push_back(lib);
    if (cudaLibraryGetKernel(&kernel, lib, j.lowered.c_str()) != cudaSuccess) {
      cudaGetLastError();
      if (log) *log = "cudaLibraryGetKernel failed for " + j.lowered;
      return false;
    }
    k->push_back(reinterpret_cast<const void *>(kernel));
  }
  return true;
}

bool device_is_sm100(std::string *log) {
  int dev = 0, major = 0, minor = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
  cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
  if (major != 10 || minor != 0) {
    if (log) *log = "runtime compilation targets sm_100a only";
    return false;
  }
  return true;
}

std::map<std::string, AdjKernels> g_adj_cache;

}  // namespace

bool jit_compile(const std::string &policy_source, bool fp32, std::vector<JitKernel> *out, std::string *log) {
  const char *T = fp32 ? "float" : "double";
  const std::string src = "#include \"milne.cuh\"\n#include \"local.cuh\"\nnamespace dl {\n" + policy_source + "}\n";
  const std::vector<std::string> names = {
      std::string("&dl::k_persistent<") + T + ", dl::YieldJit, false>",
      std::string("&dl::k_element<") + T + ", dl::YieldJit, false>",
      std::string("&dl::k_node<") + T + ", false>",
      std::string("&dl::k_internal_force<") + T + ", dl::YieldJit>",
      std::string("&dl::k_gather_force<") + T + ">",
      std::string("&dl::k_persistent<") + T + ", dl::YieldJit, true>",
      std::string("&dl::k_element<") + T + ", dl::YieldJit, true>",
      std::string("&dl::k_node<") + T + ", true>",
      std::string("&dl::k_milne<") + T + ", dl::YieldJit>",
      std::string("&dl::k_persistent<") + T + ", dl::YieldJit, false, true>",
      std::string("&dl::k_local<") + T + ", dl::YieldJit, 1>",
      std::string("&dl::k_local<") + T + ", dl::YieldJit, 2>"};
  return compile_kernels(src, names, fp32, "step", out, log);
}

bool jit_compile_adjoint(const std::string &adj_policy_source, bool fp32, std::vector<JitKernel> *out,
                         std::string *log) {
  const char *T = fp32 ? "float" : "double";
  const std::string src = "#include \"adjoint_kernels.cuh\"\nnamespace dl {\n" + adj_policy_source + "}\n";
  const std::vector<std::string> names = {std::string("&dl::k_adj_node<") + T + ">",
                                          std::string("&dl::k_adj_elem<") + T + ", dl::YieldAdj>"};
  return compile_kernels(src, names, fp32, "adjoint", out, log);
}

const AdjKernels *jit_adjoint_kernels(const std::string &adj_policy_source, bool fp32, std::string *log) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (!device_is_sm100(log)) return nullptr;
  int dev = 0;
  cudaGetDevice(&dev);
  const std::string key = std::string(fp32 ? "f|" : "d|") + std::to_string(dev) + "|" + adj_policy_source;
  auto it = g_adj_cache.find(key);
  if (it != g_adj_cache.end()) return &it->second;
  std::vector<JitKernel> jk;
  std::vector<cudaLibrary_t> libs;  // loaded until the process ends
  std::vector<const void *> k;
  if (!jit_compile_adjoint(adj_policy_source, fp32, &jk, log) || !load_kernels(jk, &libs, &k, log)) return nullptr;
  AdjKernels &ak = g_adj_cache[key];
  ak.node = k[0];
  ak.elem = k[1];
  return &ak;
}

const KernelSet *jit_kernels(const std::string &policy_source, bool fp32, std::string *log) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (!device_is_sm100(log)) return nullptr;
  int dev = 0;
  cudaGetDevice(&dev);
  const std::string key = std::string(fp32 ? "f|" : "d|") + std::to_string(dev) + "|" + policy_source;
  auto it = g_cache.find(key);
  if (it != g_cache.end()) return &it->second->ks;
  std::vector<JitKernel> jk;
  std::vector<const void *> k;
  auto e = std::make_unique<Entry>();
  if (!jit_compile(policy_source, fp32, &jk, log) || !load_kernels(jk, &e->libs, &k, log)) return nullptr;
  e->ks.persistent = k[0];
  e->ks.element = k[1];
  e->ks.node = k[2];
  e->ks.internal_force = k[3];
  e->ks.gather = k[4];
  e->ks.persistent_x = k[5];
  e->ks.element_x = k[6];
  e->ks.node_x = k[7];
  e->ks.milne = k[8];
  e->ks.persistent1 = k[9];
  e->ks.local[0] = k[10];
  e->ks.local[1] = k[11];
  e->ks.local_threads = fp32 ? LocalThreads<float>::value : LocalThreads<double>::value;
  e->ks.full_threads = fp32 ? 320 : 256;  // PersistShape<T, false>::kThreads
  e->ks.full_threads_x = 256;             // PersistShape<T, true>::kThreads
  set_persistent_caps(e->ks);
  e->ks.jit = true;
  const KernelSet *out = &e->ks;
  g_cache[key] = std::move(e);
  return out;
}

}  // namespace dl
