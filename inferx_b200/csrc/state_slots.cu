// Zeroing the state of slots that new requests take over: one launch for all of a model's
// state tensors, whose addresses and slot numbers travel as kernel parameters.
//
// What counts here is the host: an index tensor made from a Python list is a copy out of
// pageable memory, which waits for everything the device still has to do, so that the layout and
// the launch of a step that opens a request found the device idle.  With it the device waited
// 180 to 290 us ahead of each prompt step of 1,100 to 2,800 us.
#include "common.cuh"

#define ZS_TENSORS 24
#define ZS_SLOTS 64
#define ZS_THREADS 256
#define ZS_BLOCK_BYTES (ZS_THREADS * 64)

struct ZeroSlots {
  unsigned char* base[ZS_TENSORS];
  unsigned long long bytes[ZS_TENSORS];      // of one slot
  int slot[ZS_SLOTS];
};

__global__ void zero_slots_kernel(const __grid_constant__ ZeroSlots z) {
  const unsigned long long bytes = z.bytes[blockIdx.y];
  const unsigned long long from = (unsigned long long)blockIdx.x * ZS_BLOCK_BYTES;
  if (from >= bytes) return;
  const unsigned long long n = min((unsigned long long)ZS_BLOCK_BYTES, bytes - from);
  unsigned char* p = z.base[blockIdx.y] + (unsigned long long)z.slot[blockIdx.z] * bytes + from;
  if ((((uintptr_t)p | n) & 15) == 0) {
    for (unsigned i = threadIdx.x * 16; i < n; i += ZS_THREADS * 16)
      *reinterpret_cast<uint4*>(p + i) = make_uint4(0, 0, 0, 0);
  } else {                                   // a few bytes a slot, or an odd size
    for (unsigned i = threadIdx.x; i < n; i += ZS_THREADS) p[i] = 0;
  }
}

// bases, bytes: host arrays of base addresses and bytes a slot; slots: host array.
IX_API int ix_zero_slots(const unsigned long long* bases, const unsigned long long* bytes,
                         int n_tensors, const int* slots, int n_slots, cudaStream_t stream) {
  for (int t0 = 0; t0 < n_tensors; t0 += ZS_TENSORS)
    for (int s0 = 0; s0 < n_slots; s0 += ZS_SLOTS) {
      ZeroSlots z = {};
      const int nt = n_tensors - t0 < ZS_TENSORS ? n_tensors - t0 : ZS_TENSORS;
      const int ns = n_slots - s0 < ZS_SLOTS ? n_slots - s0 : ZS_SLOTS;
      unsigned long long most = 0;
      for (int t = 0; t < nt; ++t) {
        z.base[t] = reinterpret_cast<unsigned char*>(bases[t0 + t]);
        z.bytes[t] = bytes[t0 + t];
        most = bytes[t0 + t] > most ? bytes[t0 + t] : most;
      }
      for (int s = 0; s < ns; ++s) z.slot[s] = slots[s0 + s];
      const unsigned long long blocks = (most + ZS_BLOCK_BYTES - 1) / ZS_BLOCK_BYTES;
      if (blocks == 0) continue;
      if (blocks > 0x7fffffffULL) return IX_ERR_SIZE;
      zero_slots_kernel<<<dim3((unsigned)blocks, nt, ns), ZS_THREADS, 0, stream>>>(z);
      const int rc = ix_launch_status();
      if (rc) return rc;
    }
  return IX_OK;
}
