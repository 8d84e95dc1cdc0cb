// zg_result.cu — the slots of zg_result.cuh.
#include "zg_result.cuh"

#include <mutex>

namespace {
constexpr int kSlots = 64;
constexpr size_t kSlotBytes = 256;
static_assert(sizeof(ZgPartial) <= kSlotBytes, "a result fits its slot");
std::mutex g_mu;
char* g_slots = nullptr;
bool g_failed = false;
uint64_t g_free = ~0ull;
}  // namespace

ZgResultSlot::ZgResultSlot() : p(nullptr) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_slots && !g_failed &&
      cudaHostAlloc((void**)&g_slots, kSlots * kSlotBytes, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    g_slots = nullptr;
    g_failed = true;
  }
  if (!g_slots || !g_free) return;
  const int i = __builtin_ctzll(g_free);
  g_free &= g_free - 1;
  p = (ZgPartial*)(g_slots + i * kSlotBytes);
}

ZgResultSlot::~ZgResultSlot() {
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_mu);
  g_free |= 1ull << (((char*)p - g_slots) / kSlotBytes);
}
