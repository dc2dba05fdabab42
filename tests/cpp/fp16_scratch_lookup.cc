// Which scratch the FP16 launcher hands its kernel when another host thread unregisters or replaces the registered buffer
// during the call.  Links the launcher's object file with stand-ins for the rest of the library and for the CUDA runtime:
// nothing is launched, the arguments of the launch are looked at.
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../llmmm_b200/csrc/pair_walk.cuh"

namespace {
int       g_reads, g_reads_before_change;  // lookups so far / lookups that still find the first buffer
llmmm::Workspace g_first, g_then;
unsigned  g_grid, g_ways;
uint8_t * g_partials, *g_counters;
bool      g_launched;
}  // namespace

namespace llmmm {
std::atomic<uint64_t> g_launches{0}, g_split_launches{0};
int set_error(int code, const char* fmt, ...)
{
  va_list ap;
  va_start(ap, fmt);
  vfprintf(stderr, fmt, ap);
  va_end(ap);
  return code;
}
const DeviceInfo* device_info()
{
  static const DeviceInfo info{0, 148, 74, nullptr};
  return &info;
}
bool make_tmap_2d(CUtensorMap*, const void*, CUtensorMapDataType, uint32_t, uint64_t, uint64_t, uint64_t, uint32_t, uint32_t, CUtensorMapSwizzle)
{
  return true;
}
SplitPlan plan_split(const DeviceInfo*, int tiles, int k_steps, int, int, int, bool)
{
  return SplitPlan{tiles, 0, 1, k_steps, tiles < 74 ? tiles : 74, nullptr, nullptr};
}
size_t split_workspace_bytes() { return WS_HEADER_BYTES + (size_t)SPLIT_MAX_PAIRS * SPLIT_SLOT_FLOATS * sizeof(float); }
Workspace registered_workspace(int) { return g_reads++ < g_reads_before_change ? g_first : g_then; }
ScopedWorkspace::ScopedWorkspace(void*, size_t): prev_bound_(false) {}
ScopedWorkspace::~ScopedWorkspace() {}
int check_workspace_arg(const void*, size_t) { return LLMMM_OK; }
}  // namespace llmmm

extern "C" {
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void*, void** args)
{
  // fp16_gemm_kernel(tm_a, tm_b, tm_c, M, N, K, ways, chunk, partials, counters, status)
  g_launched = true;
  g_grid     = config->gridDim.x;
  g_ways     = (unsigned)*static_cast<int*>(args[6]);
  g_partials = *static_cast<uint8_t**>(args[8]);
  g_counters = *static_cast<uint8_t**>(args[9]);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { abort(); }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
void**      __cudaRegisterFatBinary(void*) { return nullptr; }
void        __cudaRegisterFatBinaryEnd(void**) {}
void        __cudaUnregisterFatBinary(void**) {}
void        __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { abort(); }
}

int main()
{
  alignas(16) static uint8_t operand[16];
  const size_t               full  = llmmm::split_workspace_bytes();
  uint8_t* const             base  = reinterpret_cast<uint8_t*>(uintptr_t(1) << 40);  // (never touched)
  uint8_t* const             other = reinterpret_cast<uint8_t*>(uintptr_t(1) << 41);
  const llmmm::Workspace     big{base, full}, none{}, small{other, llmmm::WS_HEADER_BYTES}, another{other, full};
  const int                  shapes[][3] = {{256, 256, 4096}, {130, 1096, 4104}, {385, 1096, 3592}};
  int                        bad = 0, cut = 0;
  for (const auto& s : shapes) {
    const int tiles = ((s[0] + 127) / 128) * ((s[1] + 63) / 64);
    for (const llmmm::Workspace& then : {none, small, another}) {
      for (int before = 0; before < 4; ++before) {
        g_reads               = 0;
        g_reads_before_change = before;
        g_first               = big;
        g_then                = then;
        g_launched            = false;
        if ((before & 1 ? llmmm_fp16_mm_bf16 : llmmm_fp16_mm_f16)(operand, operand, operand, s[0], s[1], s[2], nullptr) != LLMMM_OK || !g_launched) {
          printf("%dx%dx%d: not launched\n", s[0], s[1], s[2]);
          return 2;
        }
        if (g_ways == 1) {
          continue;
        }
        ++cut;
        // 32 KB of partial tile per CTA, one counter per warp of a tile; both in one buffer that is large enough
        const size_t partial_bytes = (size_t)g_grid * 32768, counter_bytes = (size_t)tiles * 4 * sizeof(uint32_t);
        auto         inside = [&](const llmmm::Workspace& w) {
          uint8_t* const p = static_cast<uint8_t*>(w.ptr);
          return p != nullptr && g_partials >= p && g_partials + partial_bytes <= p + w.bytes && g_counters >= p && g_counters + counter_bytes <= p + w.bytes;
        };
        if (g_grid != tiles * g_ways || !(inside(g_first) || inside(g_then))) {
          printf("%dx%dx%d, %zu bytes after %d lookups: a cut in %u ways with partials %p, counters %p\n", s[0], s[1], s[2], then.bytes, before, g_ways,
                 (void*)g_partials, (void*)g_counters);
          ++bad;
        }
      }
    }
  }
  printf("%d launches with cut tiles, %d of them with scratch out of range\n", cut, bad);
  return bad != 0 || cut == 0;
}
