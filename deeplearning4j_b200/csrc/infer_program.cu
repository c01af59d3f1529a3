// A run of inference convolutions from one host call.  A convolutional network's forward pass is a chain of small launches (ResNet-50:
// 53 convolutions, 8 strided gathers); issued one by one from Python each cost 25 us of host time against 15 us on the device at 32
// images.  The host plans a run once per input shape (steps and buffer offsets in one workspace) and this loop issues it: about 4 us a
// step.  Buffers, weights and inputs come with every call; nothing is kept here.
#include "common.cuh"

extern "C" int dl4j_gemm(const void* A, const void* B, void* C, void* aux, const void* bias, const void* residual, int M, int N, int K,
                         long lda, long ldb, long ldc, long ld_aux, long ld_res, int a_mn, int b_mn, int fmt, int bias_fp32, int out_fp32,
                         int act, int atomic_out, int splits, float alpha, int block_n, int num_sms, void* stream_);
extern "C" int dl4j_conv2d(int mode, const void* in, const void* w_cl, void* out, const void* bias, int N, int H, int W, int Cin, int OH,
                           int OW, int Cout, int kH, int kW, int pad_h, int pad_w, int dil_h, int dil_w, int fmt, int bias_fp32, int act,
                           int fuse_w, void* stream_);
extern "C" int dl4j_subsample(const void* in, void* out, const int* shape, int backward, void* stream);
extern "C" int dl4j_add_relu(const void* a, const void* b, void* y, long long n, void* stream_);

struct InferStep {
  int kind;                    // 0 1x1 convolution, 1 k x k convolution (stride 1), 2 strided gather, 3 relu(a + b)
  int N, H, W, C, OH, OW, O, kH, kW, p0, p1, d0, d1, relu, block_n;      // gather: p0 / p1 are the strides
  long long in, res, out;      // byte offsets into the workspace; -1 - i: external buffer i; res INT64_MIN: none
  long long w, b;              // element offsets of the folded weights and biases
};

// ext: external input buffers.  Returns 0 or the first step's error code.
DL4J_API int dl4j_infer_program(const void* steps_, int n, void* workspace, void* const* ext, const void* w, const float* b, int fmt, int num_sms,
                                void* stream) {
  const InferStep* steps = reinterpret_cast<const InferStep*>(steps_);
  const long long none = (long long)(1ULL << 63);
  auto at = [&](long long off) -> char* { return off >= 0 ? reinterpret_cast<char*>(workspace) + off : reinterpret_cast<char*>(ext[-1 - off]); };
  for (int i = 0; i < n; ++i) {
    const InferStep& s = steps[i];
    const uint16_t* ws = reinterpret_cast<const uint16_t*>(w) + s.w;
    int rc = 0;
    if (s.kind == 0) {
      const bool res = s.res != none;
      rc = dl4j_gemm(at(s.in), ws, at(s.out), nullptr, b + s.b, res ? at(s.res) : nullptr, s.N * s.H * s.W, s.O, s.C, s.C, s.C, s.O, 0, s.O, 0, 0,
                     fmt, 1, 0, s.relu ? (res ? 1 << 16 : 1) : 0, 0, 1, 1.0f, s.block_n, num_sms, stream);
    } else if (s.kind == 1) {
      rc = dl4j_conv2d(0, at(s.in), ws, at(s.out), b + s.b, s.N, s.H, s.W, s.C, s.OH, s.OW, s.O, s.kH, s.kW, s.p0, s.p1, s.d0, s.d1, fmt, 1,
                       s.relu, 0, stream);
    } else if (s.kind == 2) {
      const int shape[12] = {s.N, s.H, s.W, s.C, s.OH, s.OW, 1, 1, s.p0, s.p1, 0, 0};
      rc = dl4j_subsample(at(s.in), at(s.out), shape, 0, stream);
    } else if (s.kind == 3) {
      rc = dl4j_add_relu(at(s.in), at(s.res), at(s.out), (long long)s.N * s.H * s.W * s.C, stream);
    } else {
      rc = -DL4J_ERR_BAD_ARG;
    }
    if (rc) return rc;
  }
  return 0;
}
