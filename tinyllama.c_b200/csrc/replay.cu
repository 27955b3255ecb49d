// Calls of this library made again from a table.
//
// A prompt's step makes the same dozen calls for every layer of a model whose layers are alike, with other weights and
// another part of the cache.  Each of them costs a dozen microseconds on its way through Python (checks, views, argument
// conversion) against two to three for the launch itself, which is what prompts of up to some hundred tokens consist of (24
// layers of the 1.5B sizes: 4.3 ms for 23 tokens).  The caller makes one layer's calls one by one, notes them, and
// hands the other layers' over as one table.  Every call goes through its exported function with all of that function's
// checks and choices.
#include "common.cuh"
#include <string.h>
#include <type_traits>
#include <utility>

namespace {

// An argument from its 64-bit word: pointers and integers by value, floats by their bits.
template <typename T> T from_word(unsigned long long w) {
  if constexpr (std::is_pointer<T>::value) return reinterpret_cast<T>((uintptr_t)w);
  else if constexpr (std::is_same<T, float>::value) {
    const unsigned u = (unsigned)w;
    float f;
    memcpy(&f, &u, sizeof f);
    return f;
  } else return (T)(long long)w;
}
template <auto F> struct Call;
template <typename... A, int (*F)(A...)> struct Call<F> {
  static constexpr int n = sizeof...(A);
  template <size_t... I> static int apply(const unsigned long long* w, std::index_sequence<I...>) { return F(from_word<A>(w[I])...); }
  static int run(const unsigned long long* w) { return apply(w, std::make_index_sequence<sizeof...(A)>()); }
};

struct Entry {
  const char* name;
  int n_args;
  int (*run)(const unsigned long long*);
};
#define TLC_ENTRY(f) {#f, Call<f>::n, Call<f>::run}
const Entry kEntries[] = {
    TLC_ENTRY(tlc_event_record), TLC_ENTRY(tlc_event_wait),
    TLC_ENTRY(tlc_rmsnorm), TLC_ENTRY(tlc_gated_rmsnorm), TLC_ENTRY(tlc_gated_rmsnorm_step),
    TLC_ENTRY(tlc_linear), TLC_ENTRY(tlc_linear_swiglu), TLC_ENTRY(tlc_glu),
    TLC_ENTRY(tlc_rope_kv_store), TLC_ENTRY(tlc_attention), TLC_ENTRY(tlc_attention_decode), TLC_ENTRY(tlc_attention_decode_fused),
    TLC_ENTRY(tlc_attention_prefill), TLC_ENTRY(tlc_attention_prefill_tc),
    TLC_ENTRY(tlc_mamba_conv), TLC_ENTRY(tlc_mamba_step), TLC_ENTRY(tlc_ssm_scan), TLC_ENTRY(tlc_ssm_scan_one_row), TLC_ENTRY(tlc_ssm_scan_chunked), TLC_ENTRY(tlc_ssm_scan_ssd),
};
#undef TLC_ENTRY
constexpr int kCount = (int)(sizeof(kEntries) / sizeof(kEntries[0]));

}  // namespace

extern "C" int tlc_event_record(void* event, cudaStream_t stream) {
  const cudaError_t e = cudaEventRecord((cudaEvent_t)event, stream);
  return e == cudaSuccess ? 0 : tlc_fail(-2, "event_record: %s", cudaGetErrorString(e));
}

extern "C" int tlc_event_wait(void* event, cudaStream_t stream) {
  const cudaError_t e = cudaStreamWaitEvent(stream, (cudaEvent_t)event, 0);
  return e == cudaSuccess ? 0 : tlc_fail(-2, "event_wait: %s", cudaGetErrorString(e));
}

extern "C" int tlc_replay_index(const char* name) {
  for (int i = 0; name && i < kCount; i++)
    if (strcmp(kEntries[i].name, name) == 0) return i;
  return -1;
}

extern "C" int tlc_replay(const int* functions, const unsigned long long* words, long long n_words, int n_calls, int times) {
  TLC_REQUIRE(n_calls >= 0 && times >= 0, "replay: %d calls, %d times", n_calls, times);
  long long need = 0;
  for (int c = 0; c < n_calls; c++) {
    TLC_REQUIRE(functions[c] >= 0 && functions[c] < kCount, "replay: call %d names function %d", c, functions[c]);
    need += kEntries[functions[c]].n_args;
  }
  TLC_REQUIRE(need * times == n_words, "replay: %lld words for calls that take %lld", n_words, need * times);
  for (int t = 0; t < times; t++)
    for (int c = 0; c < n_calls; c++) {
      const Entry& e = kEntries[functions[c]];
      if (const int rc = e.run(words)) return rc < 0 ? rc : tlc_fail(-1, "replay: %s answered %d", e.name, rc);
      words += e.n_args;
    }
  return 0;
}
