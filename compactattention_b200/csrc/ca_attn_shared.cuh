// Host-side pieces that the attention kernels share.
#pragma once
#include <mutex>

#include "ca_common.cuh"

namespace ca {
namespace attn {

// Tensor maps of K and V with 64-token x 64-channel boxes (128-byte swizzle).  Dimensions 1..3 are ordered by
// ascending stride; slot_of_role gives the coordinate slot (0..2) of the token, page and head coordinates.
int encode_kv_maps(const ca_attn_params* p, CUtensorMap* k_map, CUtensorMap* v_map, int (&slot_of_role)[3]);

// Held over the two launches of a call whose units are cut: the pieces pass through a workspace that every call on the
// stream uses, so another thread's call must not come between the kernel that leaves them and the one that merges them.
std::mutex& pair_mutex(cudaStream_t stream);

// Few-query-row attention (ca_attn_decode.cu): true when ca_attn_compact hands the call to it.
bool decode_applies(const ca_attn_params* p);
int launch_decode(const ca_attn_params* p, const DeviceInfo& dev, cudaStream_t stream);

}  // namespace attn
}  // namespace ca
