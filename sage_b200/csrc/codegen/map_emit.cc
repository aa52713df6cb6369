// CUDA C emitter for fused elementwise maps.
//
// Reference: compile_map (src/ops/map.rs:369-410) writes one OpenCL kernel per (expression, input
// strides, input offsets): `y[gid] = expr(x_k[idx_k])`, with each idx_k either `offset + gid` or an
// ndim-step div/mul loop whose strides are literals in the source (src/ops/core.rs:113-175).
// Here:
//   * strides, extents and offsets are kernel PARAMETERS, so one compiled kernel serves every
//     tensor with the same access pattern (the source text is the cache key, as in the reference's
//     Context::get_program, but it no longer changes with the shape);
//   * axes are collapsed before emission (unit axes dropped, axes that form one run for every
//     operand merged), so the common cases need 0-2 integer divisions per element instead of ndim;
//   * when the innermost collapsed axis is unit-stride or broadcast for every operand, each thread
//     handles 4 consecutive elements with 128-bit loads and stores.
#include "map_emit.h"

#include <cstdio>
#include <sstream>

namespace sage {

static const char *kPrelude = R"(
typedef unsigned int uint;
#define SG __device__ __forceinline__
SG float sg_abs(float x) { return fabsf(x); }
SG int sg_abs(int x) { return x < 0 ? -x : x; }
SG uint sg_abs(uint x) { return x; }
SG float sg_log(float x) { return logf(x); }
SG float sg_exp(float x) { return expf(x); }
SG float sg_sqrt(float x) { return sqrtf(x); }
SG float sg_erf(float x) { return erff(x); }
SG float sg_ceil(float x) { return ceilf(x); }
SG float sg_floor(float x) { return floorf(x); }
SG float sg_round(float x) { return roundf(x); }
SG float sg_sin(float x) { return sinf(x); }
SG float sg_sinh(float x) { return sinhf(x); }
SG float sg_cos(float x) { return cosf(x); }
SG float sg_cosh(float x) { return coshf(x); }
SG float sg_tan(float x) { return tanf(x); }
SG float sg_tanh(float x) { return tanhf(x); }
SG float sg_asin(float x) { return asinf(x); }
SG float sg_asinh(float x) { return asinhf(x); }
SG float sg_acos(float x) { return acosf(x); }
SG float sg_acosh(float x) { return acoshf(x); }
SG float sg_atan(float x) { return atanf(x); }
SG float sg_atanh(float x) { return atanhf(x); }
SG float sg_square(float x) { return x * x; }
SG int sg_square(int x) { return x * x; }
SG uint sg_square(uint x) { return x * x; }
SG float sg_recip(float x) { return 1.0f / x; }
SG int sg_recip(int x) { return 1 / x; }
SG uint sg_recip(uint x) { return 1u / x; }
SG float sg_sign(float x) { return x > 0.0f ? 1.0f : (x < 0.0f ? -1.0f : (x == x ? x : 0.0f)); }
SG int sg_sign(int x) { return (x > 0) - (x < 0); }
SG uint sg_sign(uint x) { return x > 0u; }
SG float sg_pow(float a, float b) { return powf(a, b); }
SG float sg_mod(float a, float b) { return fmodf(a, b); }
SG int sg_mod(int a, int b) { return a % b; }
SG uint sg_mod(uint a, uint b) { return a % b; }
SG float sg_min(float a, float b) { return fminf(a, b); }
SG int sg_min(int a, int b) { return a < b ? a : b; }
SG uint sg_min(uint a, uint b) { return a < b ? a : b; }
SG float sg_max(float a, float b) { return fmaxf(a, b); }
SG int sg_max(int a, int b) { return a > b ? a : b; }
SG uint sg_max(uint a, uint b) { return a > b ? a : b; }
SG float sg_lit(uint bits) { return __uint_as_float(bits); }
// hi = x rounded to tf32 (nearest, ties away), lo = x - hi; when the rounding overflows or x is inf / nan,
// hi is the truncated value and lo what is left of a finite x (the rule of the GEMM's own split pass)
SG void sg_split_tf32(float x, float *hi, float *lo) {
  const uint xb = __float_as_uint(x);
  const uint hb = (xb + 0x1000u) & 0xffffe000u;  // cvt.rna.tf32.f32 of a finite value, as an add and a mask
  const bool finite = (xb & 0x7f800000u) != 0x7f800000u;
  const bool overflow = !finite || (hb & 0x7f800000u) == 0x7f800000u;
  const float hf = __uint_as_float(overflow ? (xb & 0xffffe000u) : hb);
  *hi = hf;
  *lo = finite ? x - hf : 0.f;
}
)";

// The half-precision pieces of four neighbouring results; 16 lanes hold a group of 64 (the rule of the GEMM's own split)
static const char *kPreludeH2 = R"(
SG uint sg_h2_bits(float x) { const uint b = __float_as_uint(x) & 0x7fffffffu; return b < 0x7f800000u ? b : 0u; }
SG void sg_h2_two(float x0, float x1, float f, uint *hi, uint *lo) {
  const float s0 = x0 * f, s1 = x1 * f;
  uint h, l;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(s1), "f"(s0));
  float f0, f1;
  asm("{.reg .f16 a, b; mov.b32 {a, b}, %2; cvt.f32.f16 %0, a; cvt.f32.f16 %1, b;}" : "=f"(f0), "=f"(f1) : "r"(h));
  const float r0 = sg_h2_bits(x0) == 0u ? 0.f : (s0 - f0) * 2048.f, r1 = sg_h2_bits(x1) == 0u ? 0.f : (s1 - f1) * 2048.f;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(r1), "f"(r0));
  *hi = h; *lo = l;
}
SG void sg_h2_store(float4 r, unsigned long long g, unsigned short *h2, long long plane, float *scale, float *marked) {
  uint b = sg_h2_bits(r.x);
  uint t = sg_h2_bits(r.y); b = b > t ? b : t;
  t = sg_h2_bits(r.z); b = b > t ? b : t;
  t = sg_h2_bits(r.w); b = b > t ? b : t;
  for (int o = 8; o > 0; o >>= 1) { t = __shfl_xor_sync(0xffffu << (threadIdx.x & 16), b, o); b = b > t ? b : t; }
  int e = (int)(b >> 23); e = e < 27 ? 27 : e;
  const float f = __uint_as_float((uint)(268 - e) << 23);
  uint2 hi, lo;
  sg_h2_two(r.x, r.y, f, &hi.x, &lo.x);
  sg_h2_two(r.z, r.w, f, &hi.y, &lo.y);
  *reinterpret_cast<uint2 *>(h2 + g) = hi;
  *reinterpret_cast<uint2 *>(h2 + plane + g) = lo;
  if ((threadIdx.x & 15) == 0) scale[g >> 6] = __uint_as_float((uint)(e - 14) << 23);
  if (marked) {  // an element other than 0 below 2^-14 once scaled (0, inf and nan less 1 are the largest)
    b = sg_h2_bits(r.x) - 1u;
    t = sg_h2_bits(r.y) - 1u; b = b < t ? b : t;
    t = sg_h2_bits(r.z) - 1u; b = b < t ? b : t;
    t = sg_h2_bits(r.w) - 1u; b = b < t ? b : t;
    for (int o = 8; o > 0; o >>= 1) { t = __shfl_xor_sync(0xffffu << (threadIdx.x & 16), b, o); b = b < t ? b : t; }
    if ((threadIdx.x & 15) == 0) marked[g >> 6] = (b != 0xffffffffu && __uint_as_float(b + 1u) * f < 1.f / 16384.f ? -1.f : 1.f) * __uint_as_float((uint)(e - 14) << 23);
  }
}
)";

const char *map_prelude_text() { return kPrelude; }

static const char *ctype(int dt) { return dt == SAGE_F32 ? "float" : dt == SAGE_I32 ? "int" : "uint"; }
static const char *vtype(int dt) { return dt == SAGE_F32 ? "float4" : dt == SAGE_I32 ? "int4" : "uint4"; }

sage_status map_plan(const std::string &expr, const std::vector<MapOperand> &in, int out_dtype, const void *y,
                     int out_ndim, const long long *out_ext, MapPlan *plan, bool emit_source, int planes) {
    const int nin = (int)in.size();
    // ---- collapse axes
    long long ext[k::kMaxDims];
    std::vector<std::vector<long long>> str(nin);
    int nd = 0;
    long long n = 1;
    for (int i = 0; i < out_ndim; ++i) {
        n *= out_ext[i];
        if (out_ext[i] == 1) continue;
        bool merge = nd > 0;
        if (merge)
            for (int q = 0; q < nin; ++q)
                if (str[q][nd - 1] != in[q].view.str[i] * out_ext[i]) merge = false;
        if (merge) {
            ext[nd - 1] *= out_ext[i];
            for (int q = 0; q < nin; ++q) str[q][nd - 1] = in[q].view.str[i];
        } else {
            ext[nd] = out_ext[i];
            for (int q = 0; q < nin; ++q) str[q].push_back(in[q].view.str[i]);
            ++nd;
        }
    }
    if (nd == 0) {
        ext[0] = 1;
        for (int q = 0; q < nin; ++q) str[q].push_back(0);
        nd = 1;
    }
    plan->n = n;
    plan->ndim = nd;
    for (int i = 0; i < nd; ++i) plan->ext[i] = (unsigned long long)ext[i];
    plan->strides = str;

    // ---- classify operands: D direct (idx = g), S scalar broadcast, G generic strided
    std::string modes;
    std::vector<long long> dflt(nd);
    {
        long long s = 1;
        for (int i = nd - 1; i >= 0; --i) {
            dflt[i] = s;
            s *= ext[i];
        }
    }
    bool vec_ok = (ext[nd - 1] % 4 == 0) && (reinterpret_cast<uintptr_t>(y) % 16 == 0);
    for (int q = 0; q < nin; ++q) {
        bool direct = true, scalar = true;
        for (int i = 0; i < nd; ++i) {
            if (str[q][i] != dflt[i]) direct = false;
            if (str[q][i] != 0) scalar = false;
        }
        if (n == 1) direct = true;
        char m = direct ? 'D' : scalar ? 'S' : 'G';
        const bool aligned = reinterpret_cast<uintptr_t>(in[q].ptr) % 16 == 0;
        if (m == 'D' && !aligned) vec_ok = false;
        if (in[q].slices > 1) {
            if (!direct || in[q].dtype != SAGE_F32) return SAGE_ERR_INVALID;
            m = 'Z';
            if (!aligned || in[q].slice_stride % 4) vec_ok = false;
        }
        if (m == 'G') {
            const long long inner = str[q][nd - 1];
            if (inner == 1) {
                m = 'G';  // unit inner stride: vector load possible
                if (!aligned) vec_ok = false;
                for (int i = 0; i < nd - 1; ++i)
                    if (str[q][i] % 4 != 0) vec_ok = false;
            } else if (inner == 0) {
                m = 'B';  // broadcast along the inner axis: one scalar load per 4 outputs
            } else {
                m = 'X';  // arbitrary inner stride: scalar path only
                vec_ok = false;
            }
        }
        modes.push_back(m);
    }
    const int vec = vec_ok ? 4 : 1;
    plan->vec = vec;
    const bool wide = n >= (1LL << 32);
    const char *it = wide ? "unsigned long long" : "unsigned int";
    if (vec != 4 || n % 64 != 0) planes &= ~2;
    plan->planes = planes;
    plan->signature = modes + ":" + std::to_string(vec) + ":" + std::to_string(nd) + (wide ? "w" : "n") + ((planes & 1) ? "P" : "") + ((planes & 2) ? "H" : "") + ((planes & 4) ? "O" : "");
    if (!emit_source) return SAGE_OK;  // the caller already holds the kernel for this signature

    // ---- emit
    std::ostringstream s;
    s << kPrelude;
    if (planes & 2) s << kPreludeH2;
    s << "struct MapP { long long n; unsigned long long ext[" << k::kMaxDims << "]; long long str["
      << (nin > 0 ? nin : 1) << "][" << k::kMaxDims << "]; };\n";
    s << "SG " << ctype(out_dtype) << " sage_expr(";
    for (int q = 0; q < nin; ++q) s << (q ? ", " : "") << ctype(in[q].dtype) << " x" << q;
    s << ") { return (" << ctype(out_dtype) << ")(" << expr << "); }\n";
    s << "extern \"C\" __global__ void __launch_bounds__(256) sage_map(";
    for (int q = 0; q < nin; ++q) s << "const " << ctype(in[q].dtype) << " *__restrict__ x" << q << "_buf, ";
    s << ctype(out_dtype) << " *__restrict__ y, const MapP p" << ((planes & 1) ? ", float *__restrict__ hi, const long long plane" : "")
      << ((planes & 2) ? ", unsigned short *__restrict__ h2, const long long h2_plane, float *__restrict__ h2_scale, float *__restrict__ h2_marked" : "");
    for (int q = 0; q < nin; ++q)
        if (modes[q] == 'Z') s << ", const int slices" << q << ", const long long apart" << q;
    s << ") {\n";
    // launched as a programmatic dependent: wait for the kernel before this one before touching memory
    s << "  asm volatile(\"griddepcontrol.launch_dependents;\" ::: \"memory\");\n";
    s << "  asm volatile(\"griddepcontrol.wait;\" ::: \"memory\");\n";
    s << "  const " << it << " q = (" << it << ")blockIdx.x * blockDim.x + threadIdx.x;\n";
    s << "  const " << it << " g = q * " << vec << ";\n";
    s << "  if (g >= (" << it << ")p.n) return;\n";
    bool need_coords = false;
    for (char m : modes)
        if (m == 'G' || m == 'B' || m == 'X') need_coords = true;
    if (need_coords) {
        for (int q = 0; q < nin; ++q)
            if (modes[q] != 'D' && modes[q] != 'S' && modes[q] != 'Z') s << "  long long i" << q << " = 0;\n";
        s << "  { " << it << " rem = g, c;\n";
        for (int d = nd - 1; d >= 0; --d) {
            if (d == 0)
                s << "    c = rem;\n";
            else
                s << "    c = rem % (" << it << ")p.ext[" << d << "]; rem /= (" << it << ")p.ext[" << d << "];\n";
            for (int q = 0; q < nin; ++q)
                if (modes[q] != 'D' && modes[q] != 'S' && modes[q] != 'Z') s << "    i" << q << " += (long long)c * p.str[" << q << "][" << d << "];\n";
        }
        s << "  }\n";
    }
    if (vec == 1) {
        for (int q = 0; q < nin; ++q) {
            if (modes[q] == 'Z') {
                s << "  float x" << q << " = x" << q << "_buf[g];\n#pragma unroll 8\n  for (int s = 1; s < slices" << q << "; ++s) x" << q << " += x" << q << "_buf[s * apart" << q << " + g];\n";
                continue;
            }
            s << "  const " << ctype(in[q].dtype) << " x" << q << " = x" << q << "_buf[";
            if (modes[q] == 'D') s << "g";
            else if (modes[q] == 'S') s << "0";
            else s << "i" << q;
            s << "];\n";
        }
        s << "  const " << ctype(out_dtype) << " r = sage_expr(";
        for (int q = 0; q < nin; ++q) s << (q ? ", " : "") << "x" << q;
        s << ");\n";
        if (!(planes & 4)) s << "  y[g] = r;\n";
        if (planes & 1) s << "  { float h, l; sg_split_tf32(r, &h, &l); hi[g] = h; hi[plane + g] = l; }\n";
    } else {
        for (int q = 0; q < nin; ++q) {
            const char *ct = ctype(in[q].dtype);
            if (modes[q] == 'Z') {  // eight slices in flight, added in order
                s << "  float4 v" << q << " = *reinterpret_cast<const float4 *>(x" << q << "_buf + g);\n  for (int s = 1; s < slices" << q << "; s += 8) {\n    float4 t[8];\n"
                  << "#pragma unroll\n    for (int u = 0; u < 8; ++u) if (s + u < slices" << q << ") t[u] = *reinterpret_cast<const float4 *>(x" << q << "_buf + (s + u) * apart" << q << " + g);\n"
                  << "#pragma unroll\n    for (int u = 0; u < 8; ++u) if (s + u < slices" << q << ") { v" << q << ".x += t[u].x; v" << q << ".y += t[u].y; v" << q << ".z += t[u].z; v" << q << ".w += t[u].w; }\n  }\n"
                  << "  const float a" << q << "[4] = {v" << q << ".x, v" << q << ".y, v" << q << ".z, v" << q << ".w};\n";
                continue;
            }
            if (modes[q] == 'D' || modes[q] == 'G') {
                s << "  const " << vtype(in[q].dtype) << " v" << q << " = *reinterpret_cast<const " << vtype(in[q].dtype)
                  << " *>(x" << q << "_buf + " << (modes[q] == 'D' ? std::string("g") : "i" + std::to_string(q)) << ");\n";
                s << "  const " << ct << " a" << q << "[4] = {v" << q << ".x, v" << q << ".y, v" << q << ".z, v" << q << ".w};\n";
            } else {
                s << "  const " << ct << " s" << q << " = x" << q << "_buf[" << (modes[q] == 'S' ? std::string("0") : "i" + std::to_string(q))
                  << "];\n";
                s << "  const " << ct << " a" << q << "[4] = {s" << q << ", s" << q << ", s" << q << ", s" << q << "};\n";
            }
        }
        s << "  " << vtype(out_dtype) << " r;\n";
        const char *comp[4] = {"x", "y", "z", "w"};
        for (int e = 0; e < 4; ++e) {
            s << "  r." << comp[e] << " = sage_expr(";
            for (int q = 0; q < nin; ++q) s << (q ? ", " : "") << "a" << q << "[" << e << "]";
            s << ");\n";
        }
        if (!(planes & 4)) s << "  *reinterpret_cast<" << vtype(out_dtype) << " *>(y + g) = r;\n";
        if (planes & 2) s << "  sg_h2_store(r, g, h2, h2_plane, h2_scale, h2_marked);\n";
        if (planes & 1)
            s << "  { float4 h, l; sg_split_tf32(r.x, &h.x, &l.x); sg_split_tf32(r.y, &h.y, &l.y); sg_split_tf32(r.z, &h.z, &l.z); "
                 "sg_split_tf32(r.w, &h.w, &l.w);\n    *reinterpret_cast<float4 *>(hi + g) = h; *reinterpret_cast<float4 *>(hi + plane + g) = l; }\n";
    }
    s << "}\n";
    plan->source = s.str();
    return SAGE_OK;
}

struct MapPHost {
    long long n;
    unsigned long long ext[k::kMaxDims];
};

sage_status map_launch(Context &ctx, const std::string &expr, const std::vector<MapOperand> &in, int out_dtype,
                       void *y, int out_ndim, const long long *out_ext, MapCache *cache, const k::PlaneOut &out) {
    const int planes = out_dtype == SAGE_F32 ? (out.hi ? 1 : 0) | (out.h2 ? 2 : 0) | (out.only && out.hi && !out.h2 ? 4 : 0) : 0;
    MapPlan plan;
    sage_status st = map_plan(expr, in, out_dtype, y, out_ndim, out_ext, &plan, false, planes);
    if (st) return st;
    if (plan.n == 0) return SAGE_OK;
    Module *mod = nullptr;
    if (cache && cache->owner == &ctx) {
        auto it = cache->by_signature.find(plan.signature);
        if (it != cache->by_signature.end()) mod = it->second;
    }
    if (!mod) {
        st = map_plan(expr, in, out_dtype, y, out_ndim, out_ext, &plan, true, planes);  // first use: write the source
        if (st) return st;
        st = ctx.module_get(plan.source, &mod);
        if (st) return st;
        if (cache) {
            if (cache->owner != &ctx) {
                cache->by_signature.clear();
                cache->owner = &ctx;
            }
            cache->by_signature[plan.signature] = mod;
        }
    }
    const int nin = (int)in.size();
    // by-value parameter block: n, ext[8], str[nin][8]
    std::vector<long long> pb(1 + k::kMaxDims + (size_t)(nin > 0 ? nin : 1) * k::kMaxDims, 0);
    pb[0] = plan.n;
    for (int i = 0; i < plan.ndim; ++i) pb[1 + i] = (long long)plan.ext[i];
    for (int q = 0; q < nin; ++q)
        for (int i = 0; i < plan.ndim; ++i) pb[1 + k::kMaxDims + (size_t)q * k::kMaxDims + i] = plan.strides[q][i];
    std::vector<const void *> ptrs(nin);
    std::vector<void *> params;
    for (int q = 0; q < nin; ++q) {
        ptrs[q] = in[q].ptr;
        params.push_back(&ptrs[q]);
    }
    params.push_back(&y);
    params.push_back(pb.data());
    k::PlaneOut o = out;
    if (plan.planes & 1) {
        params.push_back(&o.hi);
        params.push_back(&o.plane);
    }
    if (plan.planes & 2) {
        params.push_back(&o.h2);
        params.push_back(&o.h2_plane);
        params.push_back(&o.h2_scale);
        params.push_back(&o.h2_marked);
    }
    std::vector<int> slices(nin);
    std::vector<long long> apart(nin);
    for (int q = 0; q < nin; ++q)
        if (in[q].slices > 1) {
            slices[q] = in[q].slices;
            apart[q] = in[q].slice_stride;
            params.push_back(&slices[q]);
            params.push_back(&apart[q]);
        }
    const long long chunks = (plan.n + plan.vec - 1) / plan.vec;
    const uint32_t grid[3] = {(uint32_t)((chunks + 255) / 256), 1, 1};
    const uint32_t block[3] = {256, 1, 1};
    std::string label;
    if (ctx.verbose_names) {
        label = "map{" + expr + "}n=" + std::to_string(plan.n) + ",v" + std::to_string(plan.vec) + "," + plan.signature;
        for (char &ch : label)
            if (ch == ' ') ch = '_';
    }
    st = ctx.launch(mod, "sage_map", grid, block, 0, params.data(), label.empty() ? nullptr : label.c_str(), true);
    if (!st && out.h2 && !(plan.planes & 2)) st = k::split_h2_flat(ctx, static_cast<const float *>(y), plan.n, out.h2, out.h2_plane, out.h2_scale, out.h2_marked);
    return st;
}

}  // namespace sage
