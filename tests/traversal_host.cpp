// The traversal's state machine and box tests (csrc/lucid_kernels.cuh) compiled
// for the host, for tests/test_traversal_host.py.  Nothing here loads nodes or
// triangles: the 32-byte loads are compiled out.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector_functions.h>
#include <vector_types.h>

template <class T> static inline T __ldg(const T* p) { return *p; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline int __float_as_int(float f) { int i; std::memcpy(&i, &f, 4); return i; }
static inline float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }
static inline unsigned __float_as_uint(float f) { return (unsigned)__float_as_int(f); }
static inline float __uint_as_float(unsigned i) { return __int_as_float((int)i); }
static inline int __popc(unsigned x) { return __builtin_popcount(x); }
static inline unsigned __activemask() { return 1u; }
static inline unsigned __ballot_sync(unsigned, bool p) { return p ? 1u : 0u; }
static inline void __syncwarp() {}
static inline int max(int a, int b) { return a > b ? a : b; }
static inline int min(int a, int b) { return a < b ? a : b; }
#define __device__
#define __forceinline__ inline
#define __noinline__
#define asm(...)
#include "lucid_kernels.cuh"

using namespace lucid;

// n boxes (lo, hi) against n rays (o, d), in the FMA form and in the subtraction
// form, with a traversal's reciprocal direction.
extern "C" void host_box_tests(int n, const float* o, const float* d, const float* lo, const float* hi, float tmin,
                               float tmax, unsigned char* fma_form, unsigned char* sub_form) {
    DevScene sc;
    std::memset(&sc, 0, sizeof(sc));
    sc.num_bvh_tris = 1;
    for (int k = 0; k < n; ++k) {
        const V3 O = v3(o[3 * k], o[3 * k + 1], o[3 * k + 2]), D = v3(d[3 * k], d[3 * k + 1], d[3 * k + 2]);
        const float4 a = make_float4(lo[3 * k], lo[3 * k + 1], lo[3 * k + 2], 0.0f);
        const float4 b = make_float4(hi[3 * k], hi[3 * k + 1], hi[3 * k + 2], 0.0f);
        float tn;
        Trav s;
        trav_begin<false, false>(s, sc, O, D, tmin, tmax);
        fma_form[k] = box_hit_fma(a, b, s.ooi, s.inv, tmin, tmax, tn);
        sub_form[k] = box_hit(a, b, O, s.inv, tmin, tmax, tn);
    }
}

// Pushes `pushes` entries (codes 1, 2, ...) on a query's stack and pops until
// it is done, on a stack of kStack entries followed by `canary`: the codes
// popped, in order, go to `codes`.  Returns how many; *ok as the traversal
// reports it.
template <bool ANY, class Entry>
static int push_pop(int pushes, int canary, int* codes, int* ok) {
    struct { Entry stack[kStack]; Entry beyond[64]; } mem;
    for (Entry& e : mem.beyond) std::memcpy(&e, &canary, sizeof(int));
    Trav s;
    trav_none(s);
    s.h.t = 1e30f;
    s.node = kTravPop;
    bool good = true;
    for (int k = 1; k <= pushes; ++k) {
        if constexpr (ANY) trav_push_any(s, mem.stack, k, good);
        else trav_push(s, mem.stack, k, (float)k, good);
    }
    int n = 0;
    for (;;) {
        s.node = kTravPop;
        if constexpr (ANY) trav_pop_any(s, mem.stack);
        else trav_pop(s, mem.stack);
        if (s.node == kTravDone || n >= 4 * kStack) break;
        codes[n++] = s.node;
    }
    *ok = good;
    for (Entry& e : mem.beyond)
        if (std::memcmp(&e, &canary, sizeof(int)) != 0) return -1;   // written past the stack
    return n;
}
extern "C" int host_stack_size() { return kStack; }
extern "C" int host_push_pop(int any, int pushes, int canary, int* codes, int* ok) {
    return any ? push_pop<true, int>(pushes, canary, codes, ok) : push_pop<false, int2>(pushes, canary, codes, ok);
}
