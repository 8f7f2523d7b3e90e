"""The network's backward pass when no tensor-core weight gradient takes a
decoder layer's two-part input (the upsampled channels and the skip): the
general kernel reads the whole concatenation, never the upsampled part alone.
The host code itself, run on the CPU with its kernels recorded."""
import pytest

from tests import host_source as hs

STUBS = r"""
struct dim3 { unsigned x = 1, y = 1, z = 1; dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {} };
using cudaStream_t = void*;
using __nv_bfloat16 = unsigned short;
constexpr int CT = 16, CO_T = 32, CK = 8, EPI_GRAD = 1;
bool wgrad_takes, halo_form = true, cores = true;
bool unet_tc_two_inputs() { return cores && halo_form; }
bool unet_tc_enabled() { return cores; }
unsigned grid_for(long) { return 1; }
bool whole;  // c holds the concatenation
const __nv_bfloat16 *U = (__nv_bfloat16*)64, *SKIP = (__nv_bfloat16*)128;
__nv_bfloat16* C = (__nv_bfloat16*)192;
void k_up_concat(const __nv_bfloat16* u, int Cu, const __nv_bfloat16* s, int Cs, int B, int H, int W, __nv_bfloat16* c) {
  whole = u == U && s == SKIP && c == C && Cu + Cs == 96 && B == 2 && H == 8 && W == 16;
}
int general = 0, bias_sums = 0;
void k_grad_bf16(const float*, long, int, __nv_bfloat16*, float*) { bias_sums++; }
void k_wgrad_in3(const __nv_bfloat16*, const float*, int, int, int, float*) {}
void k_conv3_wgrad(const __nv_bfloat16* x, const float*, int, int, int cin, int, float*, float* db) {
  general = x == C && whole && cin == 96 ? 1 : -1;
  bias_sums += db != nullptr;
}
void k_flip_weights(const __nv_bfloat16*, int, int, __nv_bfloat16*) {}
template <class T, int E> void k_conv3(const float*, int, int, int, const __nv_bfloat16*, const float*, int, T*, float*, const __nv_bfloat16*) {}
bool unet_tc_conv_dgrad(cudaStream_t, const __nv_bfloat16*, int, int, int, int, const __nv_bfloat16*, int, float*, int, const __nv_bfloat16*) { return true; }
"""

WGRAD = r"""
bool unet_tc_conv_wgrad(cudaStream_t, const UnetInput& in, const __nv_bfloat16*, int, int, int, int cin, int, float*) {
  return wgrad_takes && unet_tc_two_inputs() && (in.x2 == nullptr ? in.split == cin : in.split == 64);
}
"""

MAIN = r"""
int main() {
  static float buf[16];
  static Unet n;
  n.grad = n.theta = buf;
  n.theta16 = n.wflip = n.wimg_flip = n.gbf = (__nv_bfloat16*)buf;
  // after a forward pass in two parts: all is as it was; the weight gradient
  // declines; the tensor cores, or their halo form, were switched off since
  for (int k = 0; k < 4; k++) {
    wgrad_takes = k != 1;
    cores = k != 2;
    halo_form = k != 3;
    whole = false;
    general = bias_sums = 0;
    n.split[12] = true;
    n.conv_up_bwd(nullptr, 12, U, 64, SKIP, 32, C, buf, 2, 8, 16, buf);
    std::printf("%d %d %d\n", k, general, bias_sums);
  }
}
"""


def test_the_general_weight_gradient_reads_the_whole_input(tmp_path):
    header, text = hs.source("fl_unet.h"), hs.source("fl_unet.cu")
    code = STUBS + "enum { UNET_LAYERS = 15, ACT_COUNT = 21 };\n" + hs.block(header, "struct UnetLayer")
    code += "const UnetLayer kUnetLayers[UNET_LAYERS]" + hs.between(text, " = {", "};") + "};\n"
    code += hs.block(header, "struct UnetInput") + WGRAD
    code += hs.block(header, "struct Unet {").replace("std::string err;", "").replace("std::string* err", "void* err")
    code += hs.block(text, "static int dgrad_tiles(")
    for name in ("conv_up_bwd", "conv_bwd"):
        code += hs.launches_as_calls(hs.block(text, "void Unet::%s(" % name))
    out = hs.run(tmp_path, code + MAIN).splitlines()
    assert [line.split() for line in out] == [["0", "0", "1"], ["1", "1", "1"], ["2", "1", "1"], ["3", "1", "1"]]
