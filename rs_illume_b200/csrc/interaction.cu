// SurfaceInteraction reconstruction for closest hits: what Triangle::intersect
// builds after its hit test (shapes/triangle.rs:264-415) through
// SurfaceInteraction::new and set_shading_geometry (core/interaction.rs:262-339).
//
// The barycentrics are recomputed with the traversal's own watertight test
// (so b0 = e0/det is the reference's, not 1 - b1 - b2), and every expression
// rounds as the Rust source does: round-to-nearest intrinsics (no contraction), cross products in double
// (Vector3::cross, geometry/vector3.rs:67-83), normalize as v * (1/length)
// (vector3.rs:85-95), coordinate_system dividing by the length
// (vector3.rs:520-537).
// Repairs: D14 (uv determinant duv02.x*duv12.y - duv02.y*duv12.x) and D27
// (SurfaceInteraction::new keeps Shading::default(); the shading frame starts
// as the geometric one, n, dpdu, dpdv, dndu, dndv, as in pbrt).
#include <cuda_runtime.h>

#include <cstddef>
#include <memory>
#include <vector>

#include "context.h"
#include "illume_gpu.h"
#include "shapes.cuh"

namespace ilm {
namespace {

constexpr uint32_t kShadeSphere = 0xFFFFFFFFu;
enum : uint32_t { kHasN = 1, kHasS = 2, kHasUV = 4, kReverse = 8 };

struct V3 { float x, y, z; };

__device__ __forceinline__ V3 vadd(V3 a, V3 b) { return {__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)}; }
__device__ __forceinline__ V3 vsub(V3 a, V3 b) { return {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)}; }
__device__ __forceinline__ V3 vmul(float s, V3 a) { return {__fmul_rn(s, a.x), __fmul_rn(s, a.y), __fmul_rn(s, a.z)}; }
__device__ __forceinline__ V3 vneg(V3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ float vdot(V3 a, V3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float vlen2(V3 a) { return vdot(a, a); }
// Vector3::cross: products and differences in double, rounded to float
__device__ __forceinline__ V3 vcross(V3 a, V3 b) {
    double ax = a.x, ay = a.y, az = a.z, bx = b.x, by = b.y, bz = b.z;
    return {__double2float_rn(__dsub_rn(__dmul_rn(ay, bz), __dmul_rn(az, by))),
            __double2float_rn(__dsub_rn(__dmul_rn(az, bx), __dmul_rn(ax, bz))),
            __double2float_rn(__dsub_rn(__dmul_rn(ax, by), __dmul_rn(ay, bx)))};
}
__device__ __forceinline__ V3 vnormalize(V3 a) { return vmul(__fdiv_rn(1.0f, __fsqrt_rn(vlen2(a))), a); }
__device__ __forceinline__ void coordinate_system(V3 v1, V3& v2, V3& v3) {
    if (fabsf(v1.x) > fabsf(v1.y)) {
        float len = __fsqrt_rn(__fadd_rn(__fmul_rn(v1.x, v1.x), __fmul_rn(v1.z, v1.z)));
        v2 = {__fdiv_rn(-v1.z, len), 0.0f, __fdiv_rn(v1.x, len)};
    } else {
        float len = __fsqrt_rn(__fadd_rn(__fmul_rn(v1.y, v1.y), __fmul_rn(v1.z, v1.z)));
        v2 = {0.0f, __fdiv_rn(v1.z, len), __fdiv_rn(-v1.y, len)};
    }
    v3 = vcross(v1, v2);
}
// b0*a + b1*b + b2*c, summed left to right
__device__ __forceinline__ V3 interp(float b0, float b1, float b2, V3 a, V3 b, V3 c) {
    return vadd(vadd(vmul(b0, a), vmul(b1, b)), vmul(b2, c));
}

// A vertex is one 32-byte sector: its position and normal with u and v in the
// fourth words (zeros where the mesh has none).  A triangle is its vertices and
// its mesh's flags, or kShadeSphere.
struct ShadeArgs {
    const float4* vtx;   // two per vertex
    const float4* tan;
    const uint4* tri;
    uint32_t n_prims;
};

__device__ __forceinline__ V3 xyz(float4 v) { return {v.x, v.y, v.z}; }
constexpr int kSiBlock = 128;
constexpr int kSiWords = sizeof(ilm_surface_interaction) / 4;   // 44
static_assert(sizeof(ilm_surface_interaction) == 176 && kSiWords % 4 == 0, "records are 11 16-byte words");

static_assert(offsetof(ilm_surface_interaction, n) == 24 && offsetof(ilm_surface_interaction, dpdu) == 44 &&
                  offsetof(ilm_surface_interaction, shading_n) == 92 &&
                  offsetof(ilm_surface_interaction, shading_dndu) == 128 &&
                  offsetof(ilm_surface_interaction, wo) == 152 && offsetof(ilm_surface_interaction, kind) == 172,
              "the words written below");

// Record i of a 16-byte aligned array, else word by word.
template <bool kAligned, class T>
__device__ __forceinline__ T load_record(const T* p, uint64_t i) {
    T v;
    if constexpr (kAligned) {
        const uint4* src = reinterpret_cast<const uint4*>(p + i);
        uint4* dst = reinterpret_cast<uint4*>(&v);
#pragma unroll
        for (int k = 0; k < (int)(sizeof(T) / 16); ++k) dst[k] = __ldg(src + k);
    } else {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(p + i);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
        for (int k = 0; k < (int)(sizeof(T) / 4); ++k) dst[k] = __ldg(src + k);
    }
    return v;
}

// A record with no more than its primitive, distance, kind, direction and point.
__device__ __forceinline__ void put_plain(float4* rec, const ilm_hit& h, uint32_t kind, V3 wo, V3 p) {
    rec[0] = make_float4(p.x, p.y, p.z, 0.0f);
#pragma unroll
    for (int k = 1; k < 9; ++k) rec[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    rec[9] = make_float4(0.0f, 0.0f, wo.x, wo.y);
    rec[10] = make_float4(wo.z, h.t, __uint_as_float(h.prim), __uint_as_float(kind));
}

// The SurfaceInteraction of one (ray, hit) pair, written to `rec` (11 16-byte
// words) in pieces as they are known: 44 words held to the end cost the
// registers of two resident blocks.
__device__ __forceinline__ void surface_interaction(const ShadeArgs& sa, const ilm_ray& r, const ilm_hit& h,
                                                    float4* rec) {
    const V3 o{r.o[0], r.o[1], r.o[2]}, d{r.d[0], r.d[1], r.d[2]}, zero{0.0f, 0.0f, 0.0f};
    if (h.prim >= sa.n_prims) return put_plain(rec, h, ILM_SI_MISS, zero, zero);   // or a flagged traversal error
    const uint4 tv = __ldg(sa.tri + h.prim);
    if (tv.w == kShadeSphere) return put_plain(rec, h, ILM_SI_SPHERE, vneg(d), vadd(o, vmul(h.t, d)));
    const uint32_t flags = tv.w;
    // all that the record may need is asked for at once
    const float4 *va = sa.vtx + 2ull * tv.x, *vb = sa.vtx + 2ull * tv.y, *vc = sa.vtx + 2ull * tv.z;
    const float4 pa = __ldg(va), pb = __ldg(vb), pc = __ldg(vc);
    const float4 na = __ldg(va + 1), nb = __ldg(vb + 1), nc = __ldg(vc + 1);
    const V3 p0 = xyz(pa), p1 = xyz(pb), p2 = xyz(pc);
    // barycentrics of the hit, as the traversal computed them
    TriRay tr = make_tri_ray(o.x, o.y, o.z, d.x, d.y, d.z);
    float t, b0, b1, b2;
    if (!triangle_test(tr, make_float3(p0.x, p0.y, p0.z), make_float3(p1.x, p1.y, p1.z),
                       make_float3(p2.x, p2.y, p2.z), INFINITY, t, b1, b2, &b0))
        return put_plain(rec, h, ILM_SI_MISS, vneg(d), zero);   // not a hit of this triangle
    // uv parameterisation (triangle.rs:96-112; default (0,0), (1,0), (1,1))
    float uv0[2] = {0.0f, 0.0f}, uv1[2] = {1.0f, 0.0f}, uv2[2] = {1.0f, 1.0f};
    if (flags & kHasUV) {
        uv0[0] = pa.w; uv0[1] = na.w;
        uv1[0] = pb.w; uv1[1] = nb.w;
        uv2[0] = pc.w; uv2[1] = nc.w;
    }
    // partial derivatives (triangle.rs:264-292)
    const float duv02x = __fsub_rn(uv0[0], uv2[0]), duv02y = __fsub_rn(uv0[1], uv2[1]);
    const float duv12x = __fsub_rn(uv1[0], uv2[0]), duv12y = __fsub_rn(uv1[1], uv2[1]);
    const V3 dp02 = vsub(p0, p2), dp12 = vsub(p1, p2);
    const float det = __fsub_rn(__fmul_rn(duv02x, duv12y), __fmul_rn(duv02y, duv12x));
    const bool degenerate_uv = fabsf(det) < 1e-8f;
    V3 dpdu{0, 0, 0}, dpdv{0, 0, 0};
    if (!degenerate_uv) {
        const float invdet = __fdiv_rn(1.0f, det);
        dpdu = vmul(invdet, vsub(vmul(duv12y, dp02), vmul(duv02y, dp12)));
        dpdv = vmul(invdet, vadd(vmul(-duv12x, dp02), vmul(duv02x, dp12)));
    }
    if (degenerate_uv || vlen2(vcross(dpdu, dpdv)) == 0.0f) {
        const V3 ng = vcross(vsub(p2, p0), vsub(p1, p0));
        if (vlen2(ng) == 0.0f)   // degenerate triangle: the reference reports no hit
            return put_plain(rec, h, ILM_SI_MISS, vneg(d), zero);
        coordinate_system(vnormalize(ng), dpdu, dpdv);
    }
    // error bound and hit point (triangle.rs:295-305)
    const V3 perr{__fmul_rn(kGamma7, __fadd_rn(__fadd_rn(fabsf(__fmul_rn(b0, p0.x)), fabsf(__fmul_rn(b1, p1.x))),
                                             fabsf(__fmul_rn(b2, p2.x)))),
                  __fmul_rn(kGamma7, __fadd_rn(__fadd_rn(fabsf(__fmul_rn(b0, p0.y)), fabsf(__fmul_rn(b1, p1.y))),
                                             fabsf(__fmul_rn(b2, p2.y)))),
                  __fmul_rn(kGamma7, __fadd_rn(__fadd_rn(fabsf(__fmul_rn(b0, p0.z)), fabsf(__fmul_rn(b1, p1.z))),
                                             fabsf(__fmul_rn(b2, p2.z))))};
    const V3 phit = interp(b0, b1, b2, p0, p1, p2);
    rec[0] = make_float4(phit.x, phit.y, phit.z, perr.x);
    rec[1] = make_float4(perr.y, perr.z, 0.0f, 0.0f);   // n.x, n.y follow
    rec[2] = make_float4(0.0f, __fadd_rn(__fadd_rn(__fmul_rn(b0, uv0[0]), __fmul_rn(b1, uv1[0])), __fmul_rn(b2, uv2[0])),
                         __fadd_rn(__fadd_rn(__fmul_rn(b0, uv0[1]), __fmul_rn(b1, uv1[1])), __fmul_rn(b2, uv2[1])),
                         dpdu.x);                       // n.z follows
    rec[3] = make_float4(dpdu.y, dpdu.z, dpdv.x, dpdv.y);
    rec[4] = make_float4(dpdv.z, 0.0f, 0.0f, 0.0f);
    rec[9] = make_float4(0.0f, 0.0f, -d.x, -d.y);       // shading_dndv.y and .z follow
    rec[10] = make_float4(-d.z, t, __uint_as_float(h.prim), __uint_as_float((uint32_t)ILM_SI_TRIANGLE));
    const bool reverse = (flags & kReverse) != 0;   // world-space meshes: no handedness swap
    // SurfaceInteraction::new (interaction.rs:262-316) then the triangle's
    // normal override (triangle.rs:322-331)
    V3 nrm = vnormalize(vcross(dp02, dp12));
    if (reverse) nrm = vneg(nrm);
    V3 sn = nrm, sdpdu = dpdu, sdpdv = dpdv, sdndu{0, 0, 0}, sdndv{0, 0, 0};
    if (flags & (kHasN | kHasS)) {
        // shading geometry (triangle.rs:333-414)
        V3 ns = nrm;
        if (flags & kHasN) {
            V3 nn = interp(b0, b1, b2, xyz(na), xyz(nb), xyz(nc));
            if (vlen2(nn) > 0.0f) ns = vnormalize(nn);
        }
        V3 ss = vnormalize(dpdu);
        if (flags & kHasS) {
            V3 s = interp(b0, b1, b2, xyz(__ldg(sa.tan + tv.x)), xyz(__ldg(sa.tan + tv.y)), xyz(__ldg(sa.tan + tv.z)));
            if (vlen2(s) > 0.0f) ss = vnormalize(s);
        }
        V3 ts = vcross(ss, ns);
        if (vlen2(ts) > 0.0f) {
            ts = vnormalize(ts);
            ss = vcross(ts, ns);
        } else {
            coordinate_system(ns, ss, ts);
        }
        V3 dndu{0, 0, 0}, dndv{0, 0, 0};
        if (flags & kHasN) {
            const V3 n0 = xyz(na), n1 = xyz(nb), n2 = xyz(nc);
            const V3 dn1 = vsub(n0, n2), dn2 = vsub(n1, n2);
            const float det2 = __fsub_rn(__fmul_rn(duv02x, duv12y), __fmul_rn(duv02y, duv12x));
            if (fabsf(det2) < 1e-8f) {
                const V3 dn = vcross(vsub(n2, n0), vsub(n1, n0));
                if (vlen2(dn) != 0.0f) coordinate_system(dn, dndu, dndv);
            } else {
                const float inv = __fdiv_rn(1.0f, det2);
                dndu = vmul(inv, vsub(vmul(duv12y, dn1), vmul(duv02y, dn2)));
                dndv = vmul(inv, vadd(vmul(-duv12x, dn1), vmul(duv02x, dn2)));
            }
        }
        if (reverse) ts = vneg(ts);
        // set_shading_geometry(ss, ts, dndu, dndv, true) (interaction.rs:318-339)
        sn = vnormalize(vcross(ss, ts));
        if (vdot(nrm, sn) < 0.0f) nrm = vneg(nrm);
        sdpdu = ss; sdpdv = ts; sdndu = dndu; sdndv = dndv;
    }
    reinterpret_cast<float2*>(rec + 1)[1] = make_float2(nrm.x, nrm.y);
    reinterpret_cast<float*>(rec + 2)[0] = nrm.z;
    rec[5] = make_float4(0.0f, 0.0f, 0.0f, sn.x);
    rec[6] = make_float4(sn.y, sn.z, sdpdu.x, sdpdu.y);
    rec[7] = make_float4(sdpdu.z, sdpdv.x, sdpdv.y, sdpdv.z);
    rec[8] = make_float4(sdndu.x, sdndu.y, sdndu.z, sdndv.x);
    reinterpret_cast<float2*>(rec + 9)[0] = make_float2(sdndv.y, sdndv.z);
}

// One thread per (ray, hit).  The kernel streams 48 bytes in and 176 out per
// pair, so it is bound by memory; a record is 44 words, and threads that
// stored their own records wrote 4 bytes into each of 32 separate lines at a
// time (222 us for 1,048,576 pairs on a mesh with normals and uvs, 1,220 GB/s).
// Each warp therefore lays its 32 records out in shared memory (16-byte
// stores at a 176-byte stride: eight consecutive lanes touch eight different
// bank groups, since 11 is odd) and hands the 5,632 contiguous bytes to one
// bulk copy: 79 us.  What was left was the wait on four loads in a chain (hit,
// triangle, mesh flags and positions, then normals and uvs) with 20 warps an SM
// to hide it: vertices of one sector each, read at once, 67 us; the words of a
// record written as they are known, which frees the registers of three more
// blocks, 53 us (8 blocks, which spill 24 bytes; 55 at 7, 68 at 9), 4,430 GB/s of the 48
// and 176 bytes.  kAligned: rays, hits and out on 16-byte boundaries (every
// buffer a query accepts is; this entry point also takes 4-byte aligned ones,
// which are read and written word by word, the writes still coalesced).
template <bool kAligned>
__global__ void __launch_bounds__(kSiBlock, 8) k_surface_interactions(ShadeArgs sa, const ilm_ray* __restrict__ rays,
                                                                   const ilm_hit* __restrict__ hits, uint64_t n,
                                                                   ilm_surface_interaction* __restrict__ out) {
    __shared__ __align__(16) float4 s_rec[kSiBlock / 32][32 * kSiWords / 4];
    const uint32_t lane = threadIdx.x & 31u;
    float4* warp_rec = s_rec[threadIdx.x >> 5];
    const uint64_t first = (uint64_t)blockIdx.x * kSiBlock + (threadIdx.x & ~31u);   // the warp's first record
    if (first >= n) return;
    const uint32_t rows = n - first < 32u ? (uint32_t)(n - first) : 32u;
    if (lane < rows)
        surface_interaction(sa, load_record<kAligned>(rays, first + lane), load_record<kAligned>(hits, first + lane),
                            warp_rec + lane * (kSiWords / 4));
    if constexpr (kAligned) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // this lane's record, visible to the copy
        __syncwarp();
        if (lane == 0) {
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out + first),
                         "r"((uint32_t)__cvta_generic_to_shared(warp_rec)),
                         "r"(rows * (uint32_t)sizeof(ilm_surface_interaction))
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // shared memory is the block's until then
        }
    } else {
        __syncwarp();
        const uint32_t* src = reinterpret_cast<const uint32_t*>(warp_rec);
        uint32_t* dst = reinterpret_cast<uint32_t*>(out + first);
        for (uint32_t k = lane; k < rows * kSiWords; k += 32u) dst[k] = src[k];
    }
}

cudaError_t launch_interactions(const ShadeArgs& sa, const ilm_ray* rays, const ilm_hit* hits, uint64_t n,
                                ilm_surface_interaction* out, cudaStream_t s) {
    const unsigned grid = (unsigned)((n + kSiBlock - 1) / kSiBlock);
    const bool aligned = (((uintptr_t)rays | (uintptr_t)hits | (uintptr_t)out) & 15u) == 0;
    if (aligned) k_surface_interactions<true><<<grid, kSiBlock, 0, s>>>(sa, rays, hits, n, out);
    else k_surface_interactions<false><<<grid, kSiBlock, 0, s>>>(sa, rays, hits, n, out);
    return cudaGetLastError();
}

// Builds the accel's shading data from its meshes (once).
int32_t ensure_shading(ilm_context* ctx, Accel& acc) {
    ShadingData& sd = acc.shading;
    if (sd.ready) return ILM_OK;
    size_t nv = 0, nt = 0;
    bool tangents = false;
    for (ilm_mesh_id id : acc.mesh_ids) {
        auto it = ctx->meshes.find(id);
        if (it == ctx->meshes.end()) { set_error(ctx, "surface interactions: a mesh of the accel is gone"); return ILM_ERR_NOT_FOUND; }
        const Mesh& m = *it->second;
        if (!m.is_spheres) nv += m.xyz.size() / 3;
        nt += m.n_prims;
        tangents = tangents || (!m.is_spheres && !m.s.empty());
    }
    // uninitialised: every element that a triangle names is written below
    std::unique_ptr<float4[]> vtx(new float4[2 * nv + 2]), tan(new float4[tangents ? nv + 1 : 1]);
    std::unique_ptr<uint4[]> tri(new uint4[nt + 1]);
    size_t v0 = 0, t0 = 0;
    for (ilm_mesh_id id : acc.mesh_ids) {
        const Mesh& m = *ctx->meshes.find(id)->second;
        if (m.is_spheres) {
            for (uint32_t p = 0; p < m.n_prims; ++p) tri[t0++] = make_uint4(0, 0, 0, kShadeSphere);
            continue;
        }
        const size_t n = m.xyz.size() / 3;
        auto at = [](const std::vector<float>& src, size_t v, float w) {
            return src.empty() ? make_float4(0.0f, 0.0f, 0.0f, w)
                               : make_float4(src[3 * v], src[3 * v + 1], src[3 * v + 2], w);
        };
        for (size_t v = 0; v < n; ++v) {
            vtx[2 * (v0 + v)] = at(m.xyz, v, m.uv.empty() ? 0.0f : m.uv[2 * v]);
            vtx[2 * (v0 + v) + 1] = at(m.n, v, m.uv.empty() ? 0.0f : m.uv[2 * v + 1]);
        }
        for (size_t v = 0; v < n && tangents; ++v) tan[v0 + v] = at(m.s, v, 0.0f);
        const uint32_t flags = (m.n.empty() ? 0u : (uint32_t)kHasN) | (m.s.empty() ? 0u : (uint32_t)kHasS) |
                               (m.uv.empty() ? 0u : (uint32_t)kHasUV) | (m.reverse ? (uint32_t)kReverse : 0u);
        const uint32_t base = (uint32_t)v0;
        for (uint32_t p = 0; p < m.n_prims; ++p)
            tri[t0++] = make_uint4(base + m.idx[3 * p], base + m.idx[3 * p + 1], base + m.idx[3 * p + 2], flags);
        v0 += n;
    }
    cudaError_t e;
    struct Up { DeviceBuffer& b; const void* src; size_t bytes; } ups[] = {
        {sd.vtx, vtx.get(), nv * 32}, {sd.tan, tan.get(), tangents ? nv * 16 : 0}, {sd.tri, tri.get(), nt * 16}};
    for (auto& u : ups) {
        if (u.bytes == 0) continue;
        if ((e = u.b.reserve(u.bytes)) != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc(shading)");
        if ((e = cudaMemcpy(u.b.ptr, u.src, u.bytes, cudaMemcpyHostToDevice)) != cudaSuccess)
            return cuda_fail(ctx, e, "cudaMemcpy(shading)");
    }
    sd.ready = true;
    return ILM_OK;
}

}  // namespace
}  // namespace ilm

using namespace ilm;

extern "C" int32_t ilm_surface_interactions(ilm_context* ctx, ilm_accel_id accel, const ilm_ray* rays,
                                            const ilm_hit* hits, uint64_t n, ilm_surface_interaction* out,
                                            void* stream) {
    if (!ctx || (n && (!rays || !hits || !out))) return ILM_ERR_INVALID_ARGUMENT;
    if (n == 0) return ILM_OK;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return ILM_ERR_CUDA;
    Accel* acc = find_accel(ctx, accel);
    if (!acc) { set_error(ctx, "ilm_surface_interactions: unknown accel id"); return ILM_ERR_NOT_FOUND; }
    int32_t st = ensure_shading(ctx, *acc);
    if (st != ILM_OK) return st;
    PtrKind kr = classify(rays), kh = classify(hits), ko = classify(out);
    if (kr != kh || kr != ko) {
        set_error(ctx, "ilm_surface_interactions: rays, hits and output must all be host or all device memory");
        return ILM_ERR_INVALID_ARGUMENT;
    }
    const ShadingData& sd = acc->shading;
    ShadeArgs sa{static_cast<const float4*>(sd.vtx.ptr), static_cast<const float4*>(sd.tan.ptr),
                 static_cast<const uint4*>(sd.tri.ptr), acc->host.n_prims};
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
    cudaError_t e;
    if (kr == PtrKind::kDevice) {
        if ((e = launch_interactions(sa, rays, hits, n, out, s)) != cudaSuccess)
            return cuda_fail(ctx, e, "k_surface_interactions");
        return ILM_OK;
    }
    DeviceBuffer dr, dh, dout;
    if ((e = dr.reserve(n * sizeof(ilm_ray))) != cudaSuccess || (e = dh.reserve(n * sizeof(ilm_hit))) != cudaSuccess ||
        (e = dout.reserve(n * sizeof(ilm_surface_interaction))) != cudaSuccess)
        return cuda_fail(ctx, e, "cudaMalloc(surface interactions)");
    cudaMemcpyAsync(dr.ptr, rays, n * sizeof(ilm_ray), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(dh.ptr, hits, n * sizeof(ilm_hit), cudaMemcpyHostToDevice, s);
    if ((e = launch_interactions(sa, static_cast<const ilm_ray*>(dr.ptr), static_cast<const ilm_hit*>(dh.ptr), n,
                                 static_cast<ilm_surface_interaction*>(dout.ptr), s)) != cudaSuccess)
        return cuda_fail(ctx, e, "k_surface_interactions");
    cudaMemcpyAsync(out, dout.ptr, n * sizeof(ilm_surface_interaction), cudaMemcpyDeviceToHost, s);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_fail(ctx, e, "ilm_surface_interactions");
    return ILM_OK;
}
