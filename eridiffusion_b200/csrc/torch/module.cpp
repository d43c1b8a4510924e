// Python module of the native op layer (see eri_ops.h).
#include <dlfcn.h>

#include "eri_ops.h"

namespace eri_ops {
Lib L;
std::atomic<long long> g_launches{0};

namespace {
void* must(void* h, const char* name) {
  void* p = dlsym(h, name);
  TORCH_CHECK(p, "the kernel library does not export ", name);
  return p;
}
// Resolves the kernels from the library at ``path`` (already loaded by the caller: the same handle comes back).
void init(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(h, "cannot load ", path, ": ", dlerror());
#define ERI_RESOLVE(name, args) L.name = reinterpret_cast<int(*) args>(must(h, #name));
  ERI_FUNCS(ERI_RESOLVE)
#undef ERI_RESOLVE
  L.eri_gn_workspace = reinterpret_cast<long long (*)(int, int, int, int, int)>(must(h, "eri_gn_workspace"));
}
}  // namespace
}  // namespace eri_ops

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using namespace eri_ops;
  m.def("init", &init);
  m.def("launch_count", [] { return g_launches.load(); });
  m.def("linear", &linear);
  m.def("linear_pair", &linear_pair);
  m.def("linear_glu", &linear_glu);
  m.def("small_linear", &small_linear);
  m.def("small_wgrad", [](const Tensor& dy, const Tensor& x, double s) { return small_wgrad(dy, x, s, Tensor()); });
  m.def("small_dgrad", &small_dgrad);
  m.def("prepare_lora_transposes", &prepare_lora_transposes);
  m.def("invalidate_lora_transposes", &invalidate_lora_transposes);
  m.def("lora_transposed", &lora_transposed);
  m.def("norm_modulate", &norm_modulate);
  m.def("qknorm_rope_joint", &qknorm_rope_joint);
  m.def("gate_residual", &gate_residual);
  m.def("act", &act);
  m.def("glu", &glu);
  m.def("split_tokens", &split_tokens);
  m.def("attention", &attention);
  m.def("attention_qkv", &attention_qkv);
  m.def("attention_kv", &attention_kv);
  m.def("attention_wide", &attention_wide);
  m.def("attention_bias", &attention_bias);
  m.def("attention_qkv_rope", &attention_qkv_rope);
  m.def("mse_loss", &mse_loss);
  m.def("group_norm_silu", &group_norm_silu);
  m.def("add_bias", &add_bias);
  m.def("conv2d_trained", &conv2d_trained);
  m.def("upsample2x", &upsample2x);
  m.def("single_stream", &single_stream);
}
