// Stand-ins for the launchers of rib200.h that record their arguments, pointers to shapes and plans by what they point to.
// Built by tests/test_binding_host.py, which compares what arrives from the native functions with what ctypes passes.
#include "../../include/rib200.h"

#include <cstddef>
#include <cstring>
#include <string>
#include <vector>

namespace {
std::vector<unsigned char> g_record;

template <class T> void put(T value) {
  const auto *bytes = reinterpret_cast<const unsigned char *>(&value);
  g_record.insert(g_record.end(), bytes, bytes + sizeof(T));
}
template <class... T> void put_all(T... values) { (put(values), ...); }
// field by field: padding is nobody's
void put(const Rib200AttentionShape *s) {
  put_all(s->tokens, s->query_heads, s->kv_heads, s->head_dim, s->max_context_tokens, s->past_tokens);
}
void put(const Rib200QkNormRopeShape *s) {
  put_all(s->tokens, s->heads, s->head_dim, s->rotary_dim, s->position_offset, s->rope_base);
}
void put(Rib200AttentionLaunchPolicy p) { put_all(p.implementation, p.kv_cache_dtype, p.kv_cache_layout); }
void put(const Rib200OnlineDecodePlan *p) {
  put_all(p->resolved_mode, p->partition_tokens, p->split_k_threshold_tokens, p->context_bucket_tokens,
          p->active_partition_capacity);
}
void put(const Rib200GatedDeltaShape *s) {
  put_all(s->tokens, s->hidden_size, s->key_heads, s->value_heads, s->key_dim, s->value_dim, s->conv_width, s->epsilon);
}
void put(Rib200GatedDeltaLaunchPolicy p) { put_all(p.schedule, p.warps_per_block, p.transposed_boundary_state); }

template <auto> struct Stub;
template <class... A, Rib200Status (*Declared)(A...)> struct Stub<Declared> {
  static Rib200Status call(A... arguments) {
    g_record.clear();
    (put(arguments), ...);
    return Rib200Status{RIB200_STATUS_OK, nullptr};
  }
};
} // namespace

extern "C" void *stub_address(const char *name) {
#define RIB200_STUB(entry)                                \
  if (std::strcmp(name, #entry) == 0) {                   \
    return reinterpret_cast<void *>(&Stub<&entry>::call); \
  }
  RIB200_STUB(rib200_causal_attention)
  RIB200_STUB(rib200_online_attention_prefill)
  RIB200_STUB(rib200_online_attention_decode)
  RIB200_STUB(rib200_online_attention_decode_early_kv_fetch)
  RIB200_STUB(rib200_batched_decode_attention)
  RIB200_STUB(rib200_paged_decode_attention)
  RIB200_STUB(rib200_qk_norm_rope)
  RIB200_STUB(rib200_split_full_query_gate)
  RIB200_STUB(rib200_attention_prologue)
  RIB200_STUB(rib200_gated_delta)
  RIB200_STUB(rib200_gdn_core)
  RIB200_STUB(rib200_batched_gdn_decode)
#undef RIB200_STUB
  return nullptr;
}

extern "C" std::size_t stub_record(unsigned char *out, std::size_t capacity) { // and forgets it
  const std::size_t bytes = g_record.size() < capacity ? g_record.size() : capacity;
  std::memcpy(out, g_record.data(), bytes);
  g_record.clear();
  return bytes;
}
