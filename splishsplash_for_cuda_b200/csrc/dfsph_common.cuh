// dfsph_common.cuh — types, SPH kernel functions, the canonical neighbour predicate and the
// compensated sums shared by every device kernel of the DFSPH time step.
//
// Everything here is templated on the arithmetic type Real (float = product, double = the FP64
// build of the same kernels used to state each field's FP32 error).
#pragma once

#include <cstdint>
#include <utility>
#include <cuda_runtime.h>

#include "../../include/dfsph_c.h"

namespace dfsph {

// ---- programmatic dependent launch -------------------------------------------------------------
// The kernels of a time step are launched with programmatic stream serialisation: the next kernel's
// launch is processed while the previous grid's last blocks finish, instead of after the grid has
// completed (about 2 us per kernel boundary on B200). Every kernel starts with pdl_wait(), which
// blocks until the previous grid has completed and its writes are visible, so the ordering is the
// plain stream order; each block signals its dependents when it ends (PdlTrigger). The attribute is
// left off while a loop body is captured into a graph (g_pdl_off).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
struct PdlTrigger {
    __device__ __forceinline__ ~PdlTrigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
};
#define DFSPH_PDL_ENTER \
    pdl_wait();         \
    const PdlTrigger pdl_trigger_guard_ {}

inline thread_local bool g_pdl_off = false;

template <class... KArgs, class... Args>
inline void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                       Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = g_pdl_off ? 0 : 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// ---------------------------------------------------------------------------------------------
// Launch shapes. One thread per particle for the gathers (SPlisHSPlasH/DFSPH/DFSPH_define_cuda.h:6
// uses 128); 256 threads keep 8 warps per block and let the FP64 residual reduction use one shared
// array per block.
constexpr int kBlock = 256;
constexpr int kWarpsPerBlock = kBlock / 32;
// Minimum resident blocks per SM asked of the compiler for the gather kernels (register cap).
#ifndef DFSPH_MIN_BLOCKS
#define DFSPH_MIN_BLOCKS 4
#endif
constexpr int kGatherMinBlocks = DFSPH_MIN_BLOCKS;

// Divergence and pressure minimum iteration counts of the reference GPU loops
// (DFSPH_core_cuda.cu:828 and :1378).
constexpr int kMinItersV = 3;
constexpr int kMinItersP = 2;

// Jacobi coefficient threshold m_eps (DFSPH_define_cuda.h:7); compared in double as the reference
// does (float |k| promoted against the double literal 1.0e-5).
constexpr double kEps = 1.0e-5;

// Neighbour count below which a particle gets no divergence source (DFSPH_core_cuda.cu:340-351).
constexpr uint32_t kMinNeighborsForDivergence = 20;

// ---------------------------------------------------------------------------------------------
// Vector helpers.
template <class Real> struct V3 {
    Real x, y, z;
};
template <class Real> __host__ __device__ inline V3<Real> v3(Real x, Real y, Real z) { return {x, y, z}; }

template <class Real> struct Vec4Traits;
template <> struct Vec4Traits<float> { using type = float4; };
struct alignas(32) double4a { double x, y, z, w; };
template <> struct Vec4Traits<double> { using type = double4a; };
template <class Real> using Vec4 = typename Vec4Traits<Real>::type;

template <class Real> __device__ __forceinline__ Vec4<Real> ld4(const Vec4<Real>* p) { return *p; }
template <> __device__ __forceinline__ float4 ld4<float>(const float4* p) { return __ldg(p); }

// Products and dot products with fixed rounding: the compiler may contract a * b + c into an FMA or
// not, depending on the code around it; passes that must agree bit for bit use these.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
template <class Real>
__device__ __forceinline__ Real dot3(Real ax, Real ay, Real az, Real bx, Real by, Real bz) {
    return fma(az, bz, fma(ax, bx, mul_rn(ay, by)));
}

// ---------------------------------------------------------------------------------------------
// Compensated (Kahan) accumulation of FP32 sums. For double the same code runs; the compensation
// term is simply tiny.
template <class Real> struct KSum {
    Real s = Real(0), c = Real(0);
    __device__ __forceinline__ void add(Real v) {
        const Real y = v - c;
        const Real t = s + y;
        c = (t - s) - y;
        s = t;
    }
    // Adds a * b; the product enters the compensated step unrounded (one FMA).
    __device__ __forceinline__ void add_product(Real a, Real b) {
        const Real y = fma(a, b, -c);
        const Real t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ Real value() const { return s; }
};
// Neumaier's variant: exact compensation whichever operand is larger. Used for the density
// deviation rho - rho0, a sum whose terms (the rest density, the self term, ~30 neighbour terms of
// up to a few hundred kg/m^3) cancel to a value ~1e3 times smaller than themselves.
template <class Real> struct NSum {
    Real s = Real(0), c = Real(0);
    __device__ __forceinline__ void add(Real v) {
        const Real t = s + v;
        c += (fabs(s) >= fabs(v)) ? ((s - t) + v) : ((v - t) + s);
        s = t;
    }
    __device__ __forceinline__ Real value() const { return s + c; }
};
template <class Real> struct KSum3 {
    KSum<Real> x, y, z;
    __device__ __forceinline__ void add(Real a, Real b, Real d) { x.add(a); y.add(b); z.add(d); }
    __device__ __forceinline__ void add_product(Real f, Real a, Real b, Real d) {
        x.add_product(f, a);
        y.add_product(f, b);
        z.add_product(f, d);
    }
};

// ---------------------------------------------------------------------------------------------
// Boundary forces in 64-bit fixed point: 2^32 units per newton, +-2^31 N range. Each contribution is
// rounded once to 2^-32 N (2.3e-10 N) and added with an integer atomic, so the accumulated force is
// the same whatever the order of the additions (an FP32 atomicAdd sum is not).
constexpr double kForceScale = 4294967296.0;
__device__ __forceinline__ void add_force_fx(unsigned long long* p, double f) {
    atomicAdd(p, (unsigned long long)llrint(f * kForceScale));
}

// ---------------------------------------------------------------------------------------------
// Canonical pair predicate. The reference tests (pos_i - pos_j).squaredNorm() < H*H
// (SPlisHSPlasH/DFSPH/DFSPH_macro_cuda.h:149, squaredNorm at SPlisHSPlasH/Vector.h:137). Its
// rounding depends on how the compiler contracts x*x+y*y+z*z; this library fixes one order with
// explicit round-to-nearest intrinsics so that the device kernels and the CPU oracle decide every
// pair identically: d2 = fma(dz,dz, fma(dy,dy, dx*dx)), strict d2 < H*H.
__device__ __forceinline__ bool pair_within(float xi, float yi, float zi, float xj, float yj, float zj, float H2) {
    const float dx = __fsub_rn(xi, xj), dy = __fsub_rn(yi, yj), dz = __fsub_rn(zi, zj);
    const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
    return d2 < H2;
}
__device__ __forceinline__ bool pair_within(double xi, double yi, double zi, double xj, double yj, double zj, double H2) {
    // The FP64 build decides pairs on the FP32-rounded coordinates so that both builds use the same
    // neighbour sets (positions enter both builds as the same float values).
    return pair_within((float)xi, (float)yi, (float)zi, (float)xj, (float)yj, (float)zj, (float)H2);
}

// Cell coordinate along one axis: floor(x / H + offset), the reference's
// (pos / kernelRadius) + gridOffset followed by toFloor (DFSPH_core_cuda.cu:1839-1841,
// SPlisHSPlasH/Vector.h:157), in FP32 with an IEEE division.
__device__ __forceinline__ int cell_coord(float x, float H, int offset) {
    return (int)floorf(__fadd_rn(__fdiv_rn(x, H), (float)offset));
}
__device__ __forceinline__ int cell_coord(double x, double H, int offset) {
    return cell_coord((float)x, (float)H, offset);
}

// 30-bit Morton key of 10-bit cell coordinates (x in the lowest bit of each triple).
__host__ __device__ inline uint32_t spread_bits10(uint32_t v) {
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
__host__ __device__ inline uint32_t morton3(uint32_t x, uint32_t y, uint32_t z) {
    return spread_bits10(x) | (spread_bits10(y) << 1) | (spread_bits10(z) << 2);
}
__host__ __device__ inline uint32_t compact_bits10(uint32_t v) {
    v &= 0x09249249u;
    v = (v | (v >> 2)) & 0x030C30C3u;
    v = (v | (v >> 4)) & 0x0300F00Fu;
    v = (v | (v >> 8)) & 0x030000FFu;
    v = (v | (v >> 16)) & 0x000003FFu;
    return v;
}
constexpr uint32_t kEscapedKey = 0xFFFFFFFFu;  // sorts after every valid 30-bit Morton key

// ---------------------------------------------------------------------------------------------
// Cubic spline kernel (SPlisHSPlasH/DFSPH/SPH_kernels.h:20-100, CubicKernelPerso): W and grad W
// with support H, k = 8/(pi H^3), l = 48/(pi H^3); grad W = 0 for |r| <= 1e-6.
//   W(q)      = k (6 q^3 - 6 q^2 + 1)   for q <= 1/2,   2 k (1 - q)^3   for 1/2 < q <= 1
//   grad W(r) = l q (3 q - 2) r / (|r| H)  for q <= 1/2,  -l (1 - q)^2 r / (|r| H)  for 1/2 < q <= 1
// The reference evaluates q = |r| / H and 1 / (|r| H) with two divisions and a square root per pair;
// here one reciprocal square root of |r|^2 and the precomputed 1/H give q and 1/(|r| H) with
// multiplications only (a few ulp from the division form; the CPU oracle keeps the division form
// and the parity tests bound the difference).
template <class Real> struct Cubic {
    Real H, invH, k, l, W0;
    // 1/H^2 and k in FP64 for the density terms of the FP32 build (density_term below); unused by
    // the FP64 build.
    double ih2_d, k_d;
    static __device__ __forceinline__ float rsqrt_(float v) { return rsqrtf(v); }
    static __device__ __forceinline__ double rsqrt_(double v) { return rsqrt(v); }
    __device__ __forceinline__ Real W_of_q(Real q) const {
        if (q <= Real(1)) {
            if (q <= Real(0.5)) {
                const Real q2 = q * q;
                const Real q3 = q2 * q;
                return k * (Real(6) * q3 - Real(6) * q2 + Real(1));
            }
            const Real f = Real(1) - q;
            return k * (Real(2) * f * f * f);
        }
        return Real(0);
    }
    // |r| <= 1e-6 (tested as |r|^2 <= 1e-12, the same cut-off up to rounding) gives grad W = 0 and
    // W = W0 = W(0).
    __device__ __forceinline__ Real W(Real rx, Real ry, Real rz) const {
        const Real r2 = rx * rx + ry * ry + rz * rz;
        if (!(r2 > Real(1e-12))) return W0;
        const Real q = r2 * rsqrt_(r2) * invH;
        return W_of_q(q);
    }
    // f with grad W(r) = f r (0 for |r| <= 1e-6 and beyond the support).
    __device__ __forceinline__ Real grad_factor(Real rx, Real ry, Real rz) const {
        const Real r2 = rx * rx + ry * ry + rz * rz;
        Real f = Real(0);
        if (r2 > Real(1e-12)) {
            const Real inv_rl = rsqrt_(r2);
            const Real q = r2 * inv_rl * invH;
            if (q <= Real(1)) {
                const Real c = (q <= Real(0.5)) ? l * q * (Real(3) * q - Real(2)) : l * (-(Real(1) - q) * (Real(1) - q));
                f = c * inv_rl * invH;
            }
        }
        return f;
    }
    // The same with every rounding explicit: the compiler contracts grad_factor's multiplications and
    // additions into FMAs differently from kernel to kernel. The solver passes use this one (as pair
    // coefficients), whose bits are those the passes got when each evaluated the kernel itself; the
    // FP32 density pass keeps grad_factor for its own sums for the same reason, because the sign of its
    // divergence source switches the warm start of a particle on or off.
    __device__ __forceinline__ Real pair_factor(Real rx, Real ry, Real rz) const {
        Real w;
        return pair_factor(rx, ry, rz, w);
    }
    // And w = W(r) from the same q.
    __device__ __forceinline__ Real pair_factor(Real rx, Real ry, Real rz, Real& w) const {
        const Real r2 = dot3(rx, ry, rz, rx, ry, rz);
        const Real inv_rl = rsqrt_(r2);
        const Real q = mul_rn(mul_rn(r2, inv_rl), invH);
        w = r2 > Real(1e-12) ? W_of_q(q) : W0;
        const Real g = Real(1) - q;
        const Real c = (q <= Real(0.5)) ? mul_rn(mul_rn(l, q), fma(Real(3), q, Real(-2))) : mul_rn(l, mul_rn(-g, g));
        const Real f = mul_rn(mul_rn(c, inv_rl), invH);
        return (r2 > Real(1e-12) && q <= Real(1)) ? f : Real(0);
    }
};

// ---------------------------------------------------------------------------------------------
// Density term m_j W(r_ij) of the FP32 build, evaluated in FP64 from the FP32 distance components: the
// density deviation rho - rho0 that drives the pressure solve is ~1/40 of rho at the most compressed
// particles, and a plain FP32 term carries ~5 ulp of error (|r|^2 rounding, sqrt and the steep cubic
// amplify it), i.e. ~4e-6 relative on rho - rho0, kappa and the velocities it corrects. The FP32 build
// sums rho - rho0 in FP64 from these terms.
// q = sqrt(q2) comes from the FP32 reciprocal square root and two Newton steps (Heron's method in its
// division-free form, relative error 2^-22 -> 2^-44 -> rounding) instead of the correctly rounded FP64
// square root: density pass 219 -> 212 us at 1 M particles, 412 -> 399 us at 2 M, the stored densities of 27 k
// and 250 k particles bit for bit the same. The self term (r = 0) is m k.
__device__ __forceinline__ double density_term(const Cubic<float>& K, float rx, float ry, float rz, float m) {
    const double dx = rx, dy = ry, dz = rz;
    const double q2 = fma(dz, dz, fma(dy, dy, dx * dx)) * K.ih2_d;
    if (q2 > 1.0) return 0.0;
    double w = 1.0;        // W / k; 1 to the last bit below q2 = 1e-20
    if (q2 > 1e-20) {
        const double y = (double)rsqrtf((float)q2), hy = 0.5 * y;
        double q = q2 * y;
        q = fma(hy, fma(-q, q, q2), q);
        q = fma(hy, fma(-q, q, q2), q);
        const double f = 1.0 - q;
        w = q <= 0.5 ? fma(-6.0 * q2, f, 1.0) : 2.0 * f * (f * f);
    }
    return w * (K.k_d * (double)m);
}

// ---------------------------------------------------------------------------------------------
// Neighbour lists. A particle's list is a sequence of slots, the fluid neighbours first, then the
// boundary neighbours from the next multiple of four on; four consecutive slots of a particle form a
// group, and the groups of all particles are interleaved: group g of particle i is the uint4
// nbr[g * stride + i], so a warp reads a group with one coalesced 512-byte load. The fluid part is
// filled up to a multiple of four with the particle's own index, the boundary part with its last
// entry, so that the passes have no remainder loop.
//
// Pair coefficients. The positions do not change between a neighbour search and the position update,
// so the pass that follows the search (density_alpha_kernel) stores f(r_ij) for every slot, where
// grad W_ij = f r_ij (0 for a fill-up slot); the ~13 passes of the two solvers form grad W_ij =
// f (x_i - x_j) without evaluating the kernel again. The
// passes were bound by instruction issue and the L1 pipe, not by DRAM, so the 4 bytes per slot they
// read more cost less than the ~40 instructions they save. Measured at 1 M particles, 31 neighbours:
// residual pass 138 -> 128 us, Jacobi pass 115 -> 85 us, step 2.59 -> 2.24 ms with the neighbour
// build's and the viscosity pass's share; at 250 k 0.797 -> 0.715 ms, at 27 k 0.348 -> 0.271 ms.
__host__ __device__ inline uint32_t slot_groups(uint32_t entries) { return (entries + 3u) >> 2; }
// Elements that the arrays of fluid and boundary positions have to spare after their capacity, so that
// the neighbour build's batched loads may run past the last run.
constexpr uint32_t kScanPad = 3;
// Groups that a list of at most `cap` entries can need.
__host__ __device__ inline uint32_t group_capacity(uint32_t cap) { return (cap + 6u) / 4u; }
// Element of slot k of particle i in the interleaved table (as 4-byte words).
__host__ __device__ inline size_t slot_word(uint32_t k, uint32_t stride, uint32_t i) {
    return 4u * ((size_t)(k >> 2) * stride + i) + (k & 3u);
}

// Index and coefficient groups are read once per pass, coalesced: they go through the read-only path
// without allocating in L1 (L1::no_allocate), so that the lines they would take stay with the
// neighbours' positions and velocities, which the passes re-read from L1. The asm is volatile: a load
// hoisted out of its condition would read past the list.
__device__ __forceinline__ uint4 ld_group(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_group(const float4* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ double4a ld_group(const double4a* p) { return *p; }

template <class T> __device__ __forceinline__ auto component(const T& v, int u) {
    return u == 0 ? v.x : u == 1 ? v.y : u == 2 ? v.z : v.w;
}

// Visits the slots of the groups that hold `entries` entries from idx / coef on, B (2 or 4) at a time:
// load(u, j) issues the gathers of a batch, use(u, f) consumes them in slot order. Keeping a batch of independent
// gathers in flight per thread hides the latency that a one-at-a-time loop exposes; the next group's index
// and coefficients are loaded before this group's gathers.
// Without a coefficient table (kTable false: it does not fit the device) factor(u) forms f from the loaded
// slot, the same bits; fill-up slots get 0 as in the table.
template <int B, bool kTable, class Real, class Load, class Factor, class Use>
__device__ __forceinline__ void visit_pairs(const uint4* __restrict__ idx, const Vec4<Real>* __restrict__ coef,
                                            uint32_t stride, uint32_t entries, Load&& load, Factor&& factor, Use&& use) {
    if (!entries) return;
    uint4 j = ld_group(idx);
    if constexpr (!kTable) {
        for (uint32_t k = 0; k < entries; k += 4) {
            idx += stride;
            uint4 jn;
            if (k + 4 < entries) jn = ld_group(idx);
#pragma unroll
            for (int b = 0; b < 4; b += 2) {
                load(0, component(j, b));
                load(1, component(j, b + 1));
                use(0, k + b < entries ? factor(0) : Real(0));
                use(1, k + b + 1 < entries ? factor(1) : Real(0));
            }
            j = jn;
        }
        return;
    }
    uint32_t groups = slot_groups(entries);
    Vec4<Real> f = ld_group(coef);
    while (true) {
        idx += stride;
        coef += stride;
        const bool more = --groups != 0;
        uint4 jn;
        Vec4<Real> fn;
        if (more) {
            jn = ld_group(idx);
            fn = ld_group(coef);
        }
#pragma unroll
        for (int b = 0; b < 4; b += B) {
#pragma unroll
            for (int u = 0; u < B; ++u) load(u, component(j, b + u));
#pragma unroll
            for (int u = 0; u < B; ++u) use(u, component(f, b + u));
        }
        if (!more) break;
        j = jn;
        f = fn;
    }
}

// Visits the `entries` slots of the groups from idx on, two at a time: load(u, j), then use(u) for the
// slots that are entries (k < entries).
template <class Load, class Use>
__device__ __forceinline__ void visit_neighbors(const uint4* __restrict__ idx, uint32_t stride, uint32_t entries,
                                                Load&& load, Use&& use) {
    if (!entries) return;
    uint4 j = ld_group(idx);
    for (uint32_t k = 0; k < entries; k += 4) {
        idx += stride;
        uint4 jn;
        if (k + 4 < entries) jn = ld_group(idx);
#pragma unroll
        for (int b = 0; b < 4; b += 2) {
            load(0, component(j, b));
            load(1, component(j, b + 1));
            if (k + b < entries) use(0);
            if (k + b + 1 < entries) use(1);
        }
        j = jn;
    }
}

// ---------------------------------------------------------------------------------------------
// Per-launch parameters (passed by value). The dt history mirrors DFSPHCData
// (DFSPH_c_arrays_structure.h:343-354, updateTimeStep/onSimulationStepEnd at .cpp:1100-1118).
template <class Real> struct StepParams {
    Cubic<Real> kern;
    Real H2;              // H*H for the predicate (computed in float for both builds)
    Real density0;
    Real viscosity;
    Real gx, gy, gz;
    Real h, h_future, inv_h, inv_h_future, h_ratio_to_past, h_ratio_to_past2;
    int off_x, off_y, off_z;     // grid offset (cells)
    int dim_x, dim_y, dim_z;     // cell grid extent
    uint32_t n_fluid;
    uint32_t n_boundary;
    uint32_t nbr_stride;         // row stride of the interleaved neighbour table
    uint32_t nbr_cap;            // stored neighbours per particle
    int boundary_moving;         // 1: boundary velocities are read (else zero)
    int bshift;                  // 1: the boundary translated rigidly by (bsx, bsy, bsz) since its binning
    Real bsx, bsy, bsz;
};

// Device-side control block of one solver loop (divergence or pressure).
struct LoopCtl {
    double sum;          // last residual sum over all fluid particles (FP64)
    double avg;          // sum / n
    double eta;          // tolerance (absolute)
    double init_avg;     // residual after the init pass
    int32_t iter;        // iterations done
    int32_t max_iter;
    int32_t min_iter;
    uint32_t cont;       // loop condition for the next iteration
    uint32_t ticket;     // last-block election counter
    uint32_t iter_sum;   // iterations of every loop ended since the counter was last cleared
    double aux;          // second sum of an init pass that reduces two values (learned warm start)
};

}  // namespace dfsph
