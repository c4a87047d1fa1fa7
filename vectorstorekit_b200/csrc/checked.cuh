// Device side of the CHECKED build (-DVSK_CHECKED): the range test of the kernels' global accesses.
//
// Works at source level: in a checked build the names __ldg and atomicAdd / Min / Max / Or / CAS stand for the templates
// below, which pass the address through vsk_chk_access first, and VSK_CHK(p) / VSK_CHK_W(p) do the same for a plain load /
// store (they are p itself in a normal build): `*VSK_CHK_W(out + i) = v;`.  The kernels of the few-query search, the Manhattan byte
// filter, the row lists, the int8 and product-quantised paths carry them at every global access but TMA's, whose tensor maps
// bound it.  Older kernels are tested at their read-only loads and atomics.  The function and the pointer to the range table are `static`: every module
// carries its own copy (the library is built without relocatable device code), and every module registers a setter
// with the host side (checked.cu) so that vsk_open can hand all of them the same table.
#pragma once
#ifdef VSK_CHECKED
#include <cuda_runtime.h>
#include <stdint.h>

namespace vsk {
namespace chk {

constexpr int kMaxRanges = 2048;
constexpr int kTables = 4;

struct Range {
  unsigned long long lo, hi;   // [lo, hi)
};

// Lives in device memory, one per GPU.  The host rewrites table (version + 1) % kTables and then publishes `version`:
// an access in flight keeps reading the table it started with.
struct State {
  int version;
  int count[kTables];
  unsigned long long faults;        // accesses refused so far
  unsigned long long first_addr;    // the first of them
  unsigned long long first_info;    // its size in bytes | write << 8 | misaligned << 9
  unsigned long long sink[64];      // where refused accesses go instead (a 256-byte-aligned window inside it)
  Range ranges[kTables][kMaxRanges];
};

static __device__ State* d_state = nullptr;

// Host side (checked.cu).
void register_module(void (*setter)(State*));
static void set_state(State* s) { cudaMemcpyToSymbol(d_state, &s, sizeof(s)); }
namespace {
struct ModuleRegistration {
  ModuleRegistration() { register_module(&set_state); }
};
static ModuleRegistration module_registration;
}  // namespace

// Returns `addr` when [addr, addr + bytes) lies inside a known range (or is not a global address); otherwise records
// the violation and returns the sink's address.  info = bytes | write << 8.
static __device__ __noinline__ unsigned long long vsk_chk_access(unsigned long long addr, unsigned info) {
  if (!__isGlobal(reinterpret_cast<const void*>(addr))) return addr;   // shared / local windows: bounded by hardware
  State* s = d_state;
  if (s == nullptr) return addr;                                       // no table yet (a launch before vsk_open)
  const unsigned bytes = info & 0xffu;
  const bool misaligned = (addr & (unsigned long long)(bytes - 1u)) != 0ull;   // every access size is a power of two
  // the state itself (the sink included) is always a legal target
  const unsigned long long sb = reinterpret_cast<unsigned long long>(s);
  const bool own = addr >= sb && addr + bytes <= sb + sizeof(State);
  // The first look may take the table from this SM's L1, which keeps lines of a slot that has been written again since the kernel
  // began (kTables announcements on: training that is still preparing its rows while the caller announces the next call's buffers).
  // An access is refused only by a look past L1 at a version that is still the published one after it.
  for (int look = 0; !misaligned; ++look) {
    const int v = *reinterpret_cast<volatile int*>(&s->version);
    const Range* r = s->ranges[v & (kTables - 1)];
    const int* count = &s->count[v & (kTables - 1)];
    const bool fresh = look > 0;
    int lo = 0, hi = fresh ? *reinterpret_cast<const volatile int*>(count) : *count;   // first range with r.lo > addr
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if ((fresh ? *reinterpret_cast<const volatile unsigned long long*>(&r[mid].lo) : r[mid].lo) <= addr) lo = mid + 1; else hi = mid;
    }
    if (own || (lo > 0 && addr + bytes <= (fresh ? *reinterpret_cast<const volatile unsigned long long*>(&r[lo - 1].hi) : r[lo - 1].hi)))
      return addr;
    if (fresh && (v == *reinterpret_cast<volatile int*>(&s->version) || look == 64)) break;
  }
  if (atomicAdd(&s->faults, 1ull) == 0ull) {
    s->first_addr = addr;
    s->first_info = (unsigned long long)info | (misaligned ? 0x200ull : 0ull);
  }
  return (reinterpret_cast<unsigned long long>(&s->sink[0]) + 255ull) & ~255ull;
}

template <typename T>
static __device__ __forceinline__ T* at(T* p, unsigned flags = 0u) {
  return reinterpret_cast<T*>(vsk_chk_access(reinterpret_cast<unsigned long long>(p), (unsigned)sizeof(T) | flags));
}
template <typename T>
static __device__ __forceinline__ T load(const T* p) {
  return __ldg(at(p));
}
#define VSK_CHK_ATOMIC(name, op)                              \
  template <typename T, typename V>                           \
  static __device__ __forceinline__ T name(T* p, V v) {       \
    return op(at(p, 0x100u), static_cast<T>(v));              \
  }
VSK_CHK_ATOMIC(atomic_add, atomicAdd)
VSK_CHK_ATOMIC(atomic_min, atomicMin)
VSK_CHK_ATOMIC(atomic_max, atomicMax)
VSK_CHK_ATOMIC(atomic_or, atomicOr)
#undef VSK_CHK_ATOMIC
template <typename T, typename C, typename V>
static __device__ __forceinline__ T atomic_cas(T* p, C c, V v) {
  return atomicCAS(at(p, 0x100u), static_cast<T>(c), static_cast<T>(v));
}

}  // namespace chk
}  // namespace vsk

#define __ldg(...) ::vsk::chk::load(__VA_ARGS__)
#define atomicAdd(...) ::vsk::chk::atomic_add(__VA_ARGS__)
#define atomicMin(...) ::vsk::chk::atomic_min(__VA_ARGS__)
#define atomicMax(...) ::vsk::chk::atomic_max(__VA_ARGS__)
#define atomicOr(...) ::vsk::chk::atomic_or(__VA_ARGS__)
#define atomicCAS(...) ::vsk::chk::atomic_cas(__VA_ARGS__)
#define VSK_CHK(p) (::vsk::chk::at(p))
#define VSK_CHK_W(p) (::vsk::chk::at(p, 0x100u))
#else
#define VSK_CHK(p) (p)
#define VSK_CHK_W(p) (p)
#endif  // VSK_CHECKED
