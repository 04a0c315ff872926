// Fused pointwise chains: one kernel evaluates a short straight-line program (up to 32 instructions over up to 6 input
// tensors, scalars as literals) per output element, so a chain of elementwise ops reads each input once and writes one
// output instead of one round trip through HBM per op.
//
// This is the device half of compile pass 4. The reference generates WGSL source per chain at run time and registers it
// with its runtime (omarchy_mac_torch/compile.py:256-336, csrc/fused.cpp:139-170); kernels here are compiled ahead of
// time, so the chain arrives as a program for a fixed interpreter kernel instead. The interpreter keeps its values in
// shared memory, one column per thread (dynamic register indices would go to local memory), and every thread runs the
// same instruction stream, so decoding is uniform across the block.
#include <mutex>

#include "common.cuh"

namespace omt {

constexpr int PW_THREADS = 256;
constexpr int PW_VALUES = OMT_PW_MAX_INPUTS + OMT_PW_MAX_INSTR;  // value slots: inputs first, then one per instruction

struct PwArgs {
  OmtPwProgram prog;
  const float* in[OMT_PW_MAX_INPUTS];
  int64_t stride[OMT_PW_MAX_INPUTS][8];  // element strides per output dimension (0 where the input broadcasts)
  int64_t ostride[8];
  int32_t shape[8];
  int32_t rank, n_in;
  uint32_t same;  // bit k: input k has exactly the output's strides (offset = the output's)
  int32_t out_dense;  // the output's strides are those of a dense tensor enumerated in memory order: offset = linear index
  int64_t numel;
  float* out;
};

__device__ __forceinline__ float pw_powf(float x, float p) {  // aten.pow.Tensor_Scalar for the exponents a chain carries
  if (p == 2.f) return x * x;
  if (p == 1.f) return x;
  if (p == 0.5f) return sqrtf(x);
  if (p == 0.f) return 1.f;
  return powf(x, p);
}

__device__ __forceinline__ float pw_eval(int op, float a, float b, float c) {
  switch (op) {
    case OMT_PW_ADD: return a + c * b;            // a + alpha * b
    case OMT_PW_SUB: return a - c * b;
    case OMT_PW_RSUB: return b - c * a;           // rsub(a, b, alpha) = b - alpha * a
    case OMT_PW_MUL: return a * b;
    case OMT_PW_DIV: return a / b;
    case OMT_PW_NEG: return -a;
    case OMT_PW_RELU: return fmaxf(a, 0.f);
    case OMT_PW_EXP: return expf(a);
    case OMT_PW_LOG: return logf(a);
    case OMT_PW_SQRT: return sqrtf(a);
    case OMT_PW_RSQRT: return rsqrtf(a);
    case OMT_PW_RECIP: return 1.f / a;
    case OMT_PW_ABS: return fabsf(a);
    case OMT_PW_TANH: return tanhf(a);
    case OMT_PW_SIGMOID: return 1.f / (1.f + expf(-a));
    case OMT_PW_SILU: return a / (1.f + expf(-a));
    case OMT_PW_MAX: return (a != a || b != b) ? a + b : fmaxf(a, b);  // NaN propagates like aten.maximum
    case OMT_PW_MIN: return (a != a || b != b) ? a + b : fminf(a, b);
    case OMT_PW_POW: return pw_powf(a, b);
    case OMT_PW_THRESHOLD_BWD: return b > c ? a : 0.f;                 // threshold_backward(grad, self, threshold)
    case OMT_PW_SIGMOID_BWD: return a * b * (1.f - b);                 // (grad, output)
    case OMT_PW_TANH_BWD: return a * (1.f - b * b);
    case OMT_PW_SILU_BWD: { const float s = 1.f / (1.f + expf(-b)); return a * s * (1.f + b * (1.f - s)); }
    case OMT_PW_GELU: return 0.5f * a * (1.f + erff(a * 0.70710678118654752f));
    case OMT_PW_GELU_TANH: { const float k = 0.7978845608028654f * (a + 0.044715f * a * a * a); return 0.5f * a * (1.f + tanhf(k)); }
    case OMT_PW_GELU_BWD: return a * (0.5f * (1.f + erff(b * 0.70710678118654752f)) + b * 0.3989422804014327f * expf(-0.5f * b * b));
    case OMT_PW_GELU_TANH_BWD: {
      const float k = 0.7978845608028654f * (b + 0.044715f * b * b * b), t = tanhf(k);
      return a * (0.5f * (1.f + t) + 0.5f * b * (1.f - t * t) * 0.7978845608028654f * (1.f + 0.134145f * b * b));
    }
    case OMT_PW_CLAMP: return fminf(fmaxf(a, b), c);                   // (x, lo, hi); NaN x stays NaN: fmaxf/fminf return the other operand
    case OMT_PW_HARDSWISH: return a * fminf(fmaxf(a + 3.f, 0.f), 6.f) * (1.f / 6.f);
    case OMT_PW_HARDSWISH_BWD: return b < -3.f ? 0.f : (b <= 3.f ? a * (b * (1.f / 3.f) + 0.5f) : a);  // (grad, self)
    case OMT_PW_HARDSIGMOID: return fminf(fmaxf(a + 3.f, 0.f), 6.f) * (1.f / 6.f);
    case OMT_PW_HARDSIGMOID_BWD: return (b > -3.f && b < 3.f) ? a * (1.f / 6.f) : 0.f;
    default: return a;
  }
}

__global__ void __launch_bounds__(PW_THREADS) pointwise_kernel(const __grid_constant__ PwArgs a) {
  pdl_wait();
  __shared__ float val[PW_VALUES][PW_THREADS];
  const int tid = threadIdx.x;
  const int64_t i = (int64_t)blockIdx.x * PW_THREADS + tid;
  if (i >= a.numel) return;
  // offset of output element i (linear over the logical shape) and of each input
  int64_t oo = 0, off[OMT_PW_MAX_INPUTS];
#pragma unroll
  for (int k = 0; k < OMT_PW_MAX_INPUTS; k++) off[k] = 0;
  const bool all_same = a.out_dense && a.same == (1u << a.n_in) - 1u;
  if (all_same) {
    oo = i;  // every tensor has the output's dense layout: walk memory linearly
#pragma unroll
    for (int k = 0; k < OMT_PW_MAX_INPUTS; k++) off[k] = i;
  } else {
    int64_t rem = i;
    for (int d = a.rank - 1; d >= 0; d--) {
      const int64_t c = rem % a.shape[d];
      rem /= a.shape[d];
      oo += c * a.ostride[d];
#pragma unroll
      for (int k = 0; k < OMT_PW_MAX_INPUTS; k++)
        if (k < a.n_in) off[k] += c * a.stride[k][d];
    }
  }
#pragma unroll
  for (int k = 0; k < OMT_PW_MAX_INPUTS; k++)
    if (k < a.n_in) val[k][tid] = __ldg(a.in[k] + off[k]);
  float r = 0.f;
  for (int j = 0; j < a.prog.n_instr; j++) {
    const OmtPwInstr ins = a.prog.instr[j];
    float v[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const int32_t o = q == 0 ? ins.a : (q == 1 ? ins.b : ins.c);
      v[q] = o >= 0 ? val[o][tid] : a.prog.literal[-1 - o];  // >= 0: a value slot; < 0: literal number -1 - o
    }
    r = pw_eval(ins.op, v[0], v[1], v[2]);
    val[OMT_PW_MAX_INPUTS + j][tid] = r;
  }
  a.out[oo] = r;
}

// The same for tensors that all share the output's dense layout (residual adds, activations): the element index is the memory
// offset everywhere, so a thread takes four consecutive elements per trip of the program with 128-bit accesses and decodes each
// instruction once for the four. The value slots are the inputs and instructions that exist, in dynamic shared memory (a
// fixed 30 slots would leave room for one block); the newest value, which most instructions read, also stays in registers.
// One element per thread was bound by decoding, not by HBM: the 16 add + ReLU launches of a ResNet-50 eval pass (batch 32, 2.1 GB
// in all) took 1138 us; the pass goes from 3822 to 3157 us.
template <int OP>
__device__ __forceinline__ float4 pw_eval4(const float4& a, const float4& b, const float4& c) {
  return make_float4(pw_eval(OP, a.x, b.x, c.x), pw_eval(OP, a.y, b.y, c.y), pw_eval(OP, a.z, b.z, c.z), pw_eval(OP, a.w, b.w, c.w));
}
__device__ __forceinline__ float4 pw_eval4(int op, const float4& a, const float4& b, const float4& c) {
  switch (op) {
#define PW_CASE(N) case N: return pw_eval4<N>(a, b, c);
#define PW_CASES(N) PW_CASE(N) PW_CASE(N + 1) PW_CASE(N + 2) PW_CASE(N + 3) PW_CASE(N + 4) PW_CASE(N + 5) PW_CASE(N + 6) PW_CASE(N + 7)
    PW_CASES(0) PW_CASES(8) PW_CASES(16) PW_CASES(24)
#undef PW_CASES
#undef PW_CASE
    default: return a;
  }
}
static_assert(OMT_PW_OP_COUNT <= 32, "pw_eval4 dispatches 32 opcodes");

struct PwVecArgs {
  OmtPwProgram prog;  // operands renumbered: slot k = input k below n_in, n_in + j = instruction j
  const float* in[OMT_PW_MAX_INPUTS];
  int32_t n_in;
  int64_t numel;
  float* out;
};
constexpr int PW_VEC_THREADS = 128;
__global__ void __launch_bounds__(PW_VEC_THREADS) pointwise_vec4_kernel(const __grid_constant__ PwVecArgs a) {
  pdl_wait();
  extern __shared__ float4 slot[];  // [n_in + n_instr - 1][PW_VEC_THREADS]
  const int tid = threadIdx.x;
  const int64_t i = ((int64_t)blockIdx.x * PW_VEC_THREADS + tid) * 4;
  if (i >= a.numel) return;
  const bool whole = i + 4 <= a.numel;
  for (int k = 0; k < a.n_in; k++) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (whole) v = __ldg(reinterpret_cast<const float4*>(a.in[k] + i));
    else {
      v.x = __ldg(a.in[k] + i);
      if (i + 1 < a.numel) v.y = __ldg(a.in[k] + i + 1);
      if (i + 2 < a.numel) v.z = __ldg(a.in[k] + i + 2);
    }
    slot[k * PW_VEC_THREADS + tid] = v;
  }
  float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
  const int last = a.prog.n_instr - 1;
  for (int j = 0; j <= last; j++) {
    const OmtPwInstr ins = a.prog.instr[j];
    auto get = [&](int32_t o) -> float4 {
      if (o < 0) {
        const float l = a.prog.literal[-1 - o];
        return make_float4(l, l, l, l);
      }
      return j > 0 && o == a.n_in + j - 1 ? r : slot[o * PW_VEC_THREADS + tid];
    };
    const float4 x = get(ins.a), y = get(ins.b), z = get(ins.c);
    r = pw_eval4(ins.op, x, y, z);
    if (j + 1 < last) slot[(a.n_in + j) * PW_VEC_THREADS + tid] = r;  // (the one before the last is only read as the newest, or not at all)
  }
  if (whole) *reinterpret_cast<float4*>(a.out + i) = r;
  else {
    a.out[i] = r.x;
    if (i + 1 < a.numel) a.out[i + 1] = r.y;
    if (i + 2 < a.numel) a.out[i + 2] = r.z;
  }
}

}  // namespace omt

using namespace omt;

extern "C" int omt_pointwise(const OmtPwProgram* prog, int32_t n_inputs, const float* const* inputs, const int64_t* in_strides,
                             const int64_t* out_strides, const int32_t* shape, int32_t rank, float* out, omt_stream_t stream) {
  OMT_REQUIRE(prog && inputs && in_strides && out_strides && shape && out, "omt_pointwise: null pointer");
  OMT_REQUIRE(n_inputs >= 1 && n_inputs <= OMT_PW_MAX_INPUTS && rank >= 0 && rank <= 8, "omt_pointwise: 1..%d inputs, rank <= 8", OMT_PW_MAX_INPUTS);
  OMT_REQUIRE(prog->n_instr >= 1 && prog->n_instr <= OMT_PW_MAX_INSTR, "omt_pointwise: 1..%d instructions", OMT_PW_MAX_INSTR);
  for (int j = 0; j < prog->n_instr; j++) {
    const OmtPwInstr& ins = prog->instr[j];
    OMT_REQUIRE(ins.op >= 0 && ins.op < OMT_PW_OP_COUNT, "omt_pointwise: unknown op %d in instruction %d", ins.op, j);
    for (int32_t o : {ins.a, ins.b, ins.c}) {
      const bool slot = o >= 0 && (o < n_inputs || (o >= OMT_PW_MAX_INPUTS && o < OMT_PW_MAX_INPUTS + j));
      OMT_REQUIRE(slot || (o < 0 && -1 - o < OMT_PW_MAX_LITERALS), "omt_pointwise: instruction %d reads operand %d, which is not defined before it", j, o);
    }
  }
  PwArgs a{};
  a.prog = *prog; a.rank = rank; a.n_in = n_inputs; a.out = out; a.numel = 1;
  for (int d = 0; d < rank; d++) {
    OMT_REQUIRE(shape[d] > 0, "omt_pointwise: empty dimension");
    a.shape[d] = shape[d]; a.ostride[d] = out_strides[d]; a.numel *= shape[d];
  }
  // dense output enumerated in memory order when its strides are the contiguous ones; a permuted dense layout (channels-last)
  // is walked linearly too when every input shares it: then the logical index does not matter, each offset equals i
  bool contiguous = true;
  int64_t expect = 1;
  for (int d = rank - 1; d >= 0; d--) {
    if (shape[d] != 1 && out_strides[d] != expect) contiguous = false;
    expect *= shape[d];
  }
  // a permuted dense layout: the sorted strides multiply up without gaps
  bool dense = contiguous;
  if (!dense) {
    int order[8];
    for (int d = 0; d < rank; d++) order[d] = d;
    for (int x = 0; x < rank; x++)
      for (int y = x + 1; y < rank; y++)
        if (out_strides[order[y]] < out_strides[order[x]]) { int t = order[x]; order[x] = order[y]; order[y] = t; }
    dense = true;
    int64_t e = 1;
    for (int x = 0; x < rank; x++) {
      const int d = order[x];
      if (shape[d] == 1) continue;
      if (out_strides[d] != e) { dense = false; break; }
      e *= shape[d];
    }
  }
  a.out_dense = dense ? 1 : 0;
  for (int k = 0; k < n_inputs; k++) {
    OMT_REQUIRE(inputs[k], "omt_pointwise: null input %d", k);
    a.in[k] = inputs[k];
    bool same = true;
    for (int d = 0; d < rank; d++) {
      a.stride[k][d] = in_strides[k * 8 + d];
      if (shape[d] != 1 && a.stride[k][d] != a.ostride[d]) same = false;
    }
    if (same) a.same |= 1u << k;
  }
  // Four elements per thread pay where decoding is what a launch takes: short programs, and long ones over enough elements to fill the SMs. The
  // chain of a long program over a few elements is latency, four times as long (24 instructions, 1 to 40 000 elements: 9.2 us against
  // 6.5, 12 instructions 5.5 against 4.5; 6 instructions 4.2 against 4.4; 300 000 elements: 10.9 against 14.7 and 6.0 against 9.3).
  bool vec = dense && (prog->n_instr <= 6 || a.numel >= 1 << 17) && a.same == (1u << n_inputs) - 1u && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  for (int k = 0; k < n_inputs; k++) vec = vec && (reinterpret_cast<uintptr_t>(inputs[k]) & 15) == 0;
  if (vec) {
    PwVecArgs v{};
    v.prog = *prog; v.n_in = n_inputs; v.numel = a.numel; v.out = out;
    for (int k = 0; k < n_inputs; k++) v.in[k] = inputs[k];
    for (int j = 0; j < prog->n_instr; j++)
      for (int32_t* o : {&v.prog.instr[j].a, &v.prog.instr[j].b, &v.prog.instr[j].c})
        if (*o >= OMT_PW_MAX_INPUTS) *o += n_inputs - OMT_PW_MAX_INPUTS;
    // (30 slots are 60 KB: more than a kernel gets without asking)
    static std::once_flag once;
    std::call_once(once, [] {
      if (cudaFuncSetAttribute(pointwise_vec4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PW_VALUES * PW_VEC_THREADS * (int)sizeof(float4)) != cudaSuccess)
        cudaGetLastError();  // (the launch reports it)
    });
    const size_t smem = (size_t)(n_inputs + prog->n_instr) * PW_VEC_THREADS * sizeof(float4);
    launch(pointwise_vec4_kernel, (unsigned)cdiv(a.numel, 4 * PW_VEC_THREADS), PW_VEC_THREADS, smem, st(stream), v);
    return check_launch("pointwise_program");
  }
  launch(pointwise_kernel, (unsigned)cdiv(a.numel, PW_THREADS), PW_THREADS, 0, st(stream), a);
  return check_launch("pointwise_program");
}
