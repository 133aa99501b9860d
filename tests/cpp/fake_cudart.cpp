// Runs the library's host code without a GPU: this program defines the CUDA
// runtime functions that libmdgemm.so calls (an executable's symbols come
// before the shared runtime's), keeps account of what they are asked for and
// prints it.  Kernels and copies do nothing, device addresses are numbers that
// nobody reads through, an allocation beyond `capacity` fails as on a full
// device and leaves the thread's last error set, as the runtime does.
//
// argv is a list of commands:
//   capacity BYTES           device memory from here on
//   digits S D               slices and diagonals of the gemm commands from here on
//   gemm FORM P M N K        mdg_gemm with the workspace that it asks for
//   host P M N K             mdg_gemm_host, BF16 form
//   plan P M N K             mdg_plan_create, its schedule, mdg_plan_destroy
//   tune P M N K             the same with mdg_plan_tune before
//   batch P M N K            mdg_batch_create and mdg_batch_run of one problem, then
//                            with the split mode off: what the first run's launch of
//                            the grouped GEMM, replayed, finds in the second's tables
//   batched FORM P M N K     mdg_gemm_batched of one problem
//   renorm P M N K           mdg_renorm_diagonals, default digits
//   save PATH / load PATH    the tuning cache
// and prints, a line each:
//   limit KERNEL BYTES       cudaFuncAttributeMaxDynamicSharedMemorySize
//   launch KERNEL SMEM [stack=S] [pace=P dealt=D]
//   malloc BYTES / oom BYTES / free BYTES
//   replay UNIT ..           the units that the replayed launch takes, in order
//   status COMMAND STATUS [engine parts raster pace]
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "mdgemm.h"

namespace {

size_t capacity = SIZE_MAX, in_use = 0;
uintptr_t next_address = (uintptr_t)1 << 40;
cudaError_t last_error = cudaSuccess;
float last_ms = 1.0f;  // of the last diagonal GEMM launched

std::map<const void *, std::string> &kernels() {
  static std::map<const void *, std::string> m;
  return m;
}

std::map<void *, size_t> &blocks() {
  static std::map<void *, size_t> m;
  return m;
}

// the identifier of a kernel in its mangled name: ..18cross_sums_kernelE..
std::string plain_name(const std::string &mangled) {
  const size_t at = mangled.find("_GLOBAL__N__");
  size_t i = at == std::string::npos ? 2 : at;
  if (at != std::string::npos) {
    while (i < mangled.size() && i > 0 && isdigit(mangled[i - 1])) --i;
    i = at + (size_t)atoi(mangled.c_str() + i);
  }
  while (i < mangled.size() && !isdigit(mangled[i])) ++i;
  const int len = atoi(mangled.c_str() + i);
  while (i < mangled.size() && isdigit(mangled[i])) ++i;
  std::string name = mangled.substr(i, len), rest = mangled.substr(i + len);
  if (!rest.empty() && rest[0] == 'I') name += rest.substr(0, rest.find('v'));
  return name;
}

// The grouped GEMM's launches, and the words last copied to the device.
struct Grouped {
  unsigned workers;
  const int *starts, *order;
};
std::vector<Grouped> grouped;
std::map<uintptr_t, int> device_words;
bool recording = false;  // (during batch commands)

// The units that a launch's workers find there; -1: no such word was written.
std::vector<int> units_of(const Grouped &g) {
  auto word = [](const int *p) {
    const auto it = device_words.find((uintptr_t)p);
    return it == device_words.end() ? -1 : it->second;
  };
  std::vector<int> units;
  for (unsigned w = 0; w < g.workers; ++w) {
    const int first = word(g.starts + w), last = word(g.starts + w + 1);
    if (first < 0 || last < 0 || last - first > 1 << 20) return {-1};
    for (int i = first; i < last; ++i) units.push_back(word(g.order + i));
  }
  return units;
}

template <class T>
T arg(void **args, int i) {
  return *reinterpret_cast<T *>(args[i]);
}

int fake_encode(void *map) {
  std::memset(map, 0, 128);
  return 0;
}

// memory that is never touched
double *reserve(size_t doubles) {
  void *p = mmap(nullptr, doubles * 8 + 4096, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE,
                 -1, 0);
  return p == MAP_FAILED ? nullptr : reinterpret_cast<double *>(p);
}

}  // namespace

extern "C" {

void **__cudaRegisterFatBinary(void *) {
  static void *handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *fun, char *, const char *name, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {
  kernels()[fun] = plain_name(name);
}

struct CallConfiguration {
  dim3 grid, block;
  size_t smem;
  void *stream;
};
static CallConfiguration pushed;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *stream) {
  pushed = CallConfiguration{grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
  *grid = pushed.grid;
  *block = pushed.block;
  *smem = pushed.smem;
  *reinterpret_cast<void **>(stream) = pushed.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fun) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(fun));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3 grid, dim3, void **args, size_t smem,
                               cudaStream_t) {
  const std::string name = kernels()[kernel];
  std::printf("launch %s %zu", name.c_str(), smem);
  if (name == "diag_gemm_tc2_kernel") {  // two diagonals an accumulator: the fast one
    last_ms = arg<int>(args, 9) ? 1.0f : 2.0f;
    std::printf(" stack=%d pace=%d dealt=%d", arg<int>(args, 9), arg<int>(args, 15),
                arg<int>(args, 18));
  } else if (name == "diag_gemm_tc_kernel") {  // tiles of 128 columns: the fast one
    last_ms = arg<int>(args, 9) == 128 ? 1.0f : 3.0f;
  } else if (name == "diag_gemm_cross_kernel") {
    std::printf(" pace=%d dealt=%d", arg<int>(args, 16), arg<int>(args, 19));
  }
  if (name.find("grouped") != std::string::npos)
    grouped.push_back(Grouped{grid.x, arg<const int *>(args, 2), arg<const int *>(args, 3)});
  std::printf("\n");
  return cudaSuccess;
}

cudaError_t cudaFuncSetAttribute(const void *fun, enum cudaFuncAttribute, int value) {
  std::printf("limit %s %d\n", kernels()[fun].c_str(), value);
  return cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t bytes) {
  if (in_use + bytes > capacity) {
    std::printf("oom %zu\n", bytes);
    *p = nullptr;
    return last_error = cudaErrorMemoryAllocation;
  }
  std::printf("malloc %zu\n", bytes);
  *p = reinterpret_cast<void *>(next_address);
  next_address += (bytes + 4095) / 4096 * 4096;
  blocks()[*p] = bytes;
  in_use += bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  std::printf("free %zu\n", blocks()[p]);
  in_use -= blocks()[p];
  blocks().erase(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}

cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr, int) {
  *v = 152;  // multiprocessors
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp *prop, int) {
  std::memset(prop, 0, sizeof *prop);
  std::strcpy(prop->name, "fake");
  return cudaSuccess;
}
cudaError_t cudaDriverGetVersion(int *v) {
  *v = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *q) {
  *f = reinterpret_cast<void *>(fake_encode);
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                                  unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = reinterpret_cast<cudaEvent_t>(1);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = last_ms;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t bytes, enum cudaMemcpyKind kind,
                            cudaStream_t) {
  if (recording && kind == cudaMemcpyHostToDevice)
    for (size_t i = 0; i + 4 <= bytes; i += 4)
      std::memcpy(&device_words[(uintptr_t)to + i], (const char *)from + i, 4);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t,
                              enum cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void *p, const void *, size_t bytes, size_t, enum cudaMemcpyKind) {
  std::memset(p, 0, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"

int main(int argc, char **argv) {
  int at = 1;
  auto word = [&]() -> std::string { return at < argc ? argv[at++] : ""; };
  auto number = [&]() { return std::atoi(word().c_str()); };
  const double *dev = reinterpret_cast<const double *>((uintptr_t)1 << 39);
  double *dev_out = reinterpret_cast<double *>((uintptr_t)1 << 39);
  mdg_options digits = {};
  while (at < argc) {
    const std::string cmd = word();
    int status = 0;
    mdg_options o = {};
    if (cmd == "capacity") {
      capacity = std::strtoull(word().c_str(), nullptr, 10);
      continue;
    } else if (cmd == "digits") {
      digits.slices = number();
      digits.diagonals = number();
      continue;
    } else if (cmd == "save") {
      status = mdg_tune_cache_save(word().c_str());
    } else if (cmd == "load") {
      status = mdg_tune_cache_load(word().c_str());
    } else if (cmd == "gemm" || cmd == "batched") {
      const int form = number(), p = number(), m = number(), n = number(), k = number();
      const mdg_problem q{p, m, n, k, dev, dev, dev_out, k, n, n};
      if (cmd == "gemm")
        status = mdg_gemm(form, p, m, n, k, dev, k, dev, n, dev_out, n, &digits, dev_out,
                          mdg_gemm_workspace_size(form, p, m, n, k, &digits), nullptr);
      else
        status = mdg_gemm_batched(form, &q, 1, nullptr, dev_out,
                                  mdg_gemm_batched_workspace_size(form, &q, 1, nullptr), nullptr);
    } else {
      const int p = number(), m = number(), n = number(), k = number();
      if (cmd == "host") {
        status = mdg_gemm_host(MDG_FORM_SLICE_BF16, p, m, n, k, reserve((size_t)m * k * p),
                               reserve((size_t)k * n * p), reserve((size_t)m * n * p), nullptr);
      } else if (cmd == "plan" || cmd == "tune") {
        mdg_plan plan = nullptr;
        status = mdg_plan_create(MDG_FORM_SLICE_BF16, p, m, n, k, nullptr, &plan);
        if (status == 0 && cmd == "tune") status = mdg_plan_tune(plan, dev, k, dev, n, dev_out, n, nullptr);
        if (status == 0) mdg_plan_schedule(plan, &o);
        mdg_plan_destroy(plan);
      } else if (cmd == "renorm") {
        const int s = mdg_default_slices(p);
        const int *in = reinterpret_cast<const int *>(dev);
        status = mdg_renorm_diagonals(p, s, s, k, m, n, in, (long long)m * n, n, in, in, dev_out, n,
                                      nullptr);
      } else if (cmd == "batch") {
        const mdg_problem q{p, m, n, k, dev, dev, dev_out, k, n, n};
        mdg_batch batch = nullptr;
        recording = true;
        status = mdg_batch_create(&q, 1, dev_out, mdg_batch_workspace_size(&q, 1), nullptr, &batch);
        if (status == 0) status = mdg_batch_run(batch, nullptr);
        if (status == 0) status = mdg_batch_set_split(batch, 0, nullptr);
        if (status == 0) {
          std::printf("replay");
          for (int u : units_of(grouped.back())) std::printf(" %d", u);
          std::printf("\n");
        }
        recording = false;
        mdg_batch_destroy(batch);
      } else {
        std::fprintf(stderr, "unknown command %s\n", cmd.c_str());
        return 2;
      }
    }
    std::printf("status %s %d %d %d %d %d\n", cmd.c_str(), status, o.engine, o.parts, o.raster, o.pace);
  }
  return 0;
}
