// gs_ply.cu — PLY ingest: host scan of the header, device conversion of the vertex block into
// records.
//
// The reference reads scenes with wgpu-3dgs-core's Gaussians::read_from_file(path,
// GaussiansSource::Ply) (examples/simple.rs:157-160) and uploads them with Viewer::new.  Here
// the header (a few hundred bytes of text) is scanned on the host and the vertex block goes to
// the device as it is in the file; one kernel then turns each vertex into a record.
//
// Kernel layout: a CTA owns 128 consecutive vertices.  It copies their bytes (128 × stride) into
// shared memory, by 16-byte cp.async where the block is 16-byte aligned (any 128 vertices then
// start on such a boundary), else by coalesced 4-byte loads; each thread builds its record in
// registers, and the records take the vertices' place in shared memory on their way out (FP32
// records by one cp.async.bulk store, half records by coalesced 16-byte stores).
//
// What bounds it: HBM.  A record's values are defined in double (gs_convert.cuh), and in double the
// kernel took 783 us for 1M degree-3 vertices into FP32 records, all of it on the double pipe
// (about 300 operations a vertex at two per clock and SM).  Worked out in pairs of floats, with the
// double path kept for the vertices whose rounding the pairs do not settle (gs_convert_fast.cuh;
// about 0.1 % of covariances), the same bits take 87 us: 472 MB at 5.4 TB/s, 80 % of a plain copy.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_bf16.h>

#include "gs_convert_fast.cuh"
#include "gs_internal.h"

namespace gs {

constexpr uint32_t kPlyThreads = 128;
constexpr uint32_t kPlyMaxStride = 1024;

// ---- header scan --------------------------------------------------------------------------
namespace {

int ply_type_bytes(const std::string &t) {
    if (t == "char" || t == "uchar" || t == "int8" || t == "uint8") return 1;
    if (t == "short" || t == "ushort" || t == "int16" || t == "uint16") return 2;
    if (t == "int" || t == "uint" || t == "int32" || t == "uint32" || t == "float" || t == "float32") return 4;
    if (t == "double" || t == "float64") return 8;
    return 0;
}

bool is_float32(const std::string &t) { return t == "float" || t == "float32"; }

gs_status ply_fail(const char *fmt, const char *arg = "") {
    char buf[256];
    snprintf(buf, sizeof(buf), fmt, arg);
    return set_error(GS_ERR_INVALID_ARG, buf);
}

std::vector<std::string> split_ws(const std::string &line) {
    std::vector<std::string> out;
    size_t i = 0;
    while (i < line.size()) {
        while (i < line.size() && (line[i] == ' ' || line[i] == '\t' || line[i] == '\r')) ++i;
        size_t j = i;
        while (j < line.size() && !(line[j] == ' ' || line[j] == '\t' || line[j] == '\r')) ++j;
        if (j > i) out.emplace_back(line.substr(i, j - i));
        i = j;
    }
    return out;
}

bool parse_u64(const std::string &s, uint64_t *v) {
    if (s.empty() || s.size() > 19) return false;
    uint64_t x = 0;
    for (char c : s) {
        if (c < '0' || c > '9') return false;
        x = x * 10 + (uint64_t)(c - '0');
    }
    *v = x;
    return true;
}

}  // namespace

// Checks that every field offset the kernel reads lies inside a vertex.
gs_status ply_check_layout(const gs_ply_layout *L) {
    if (!L) return set_error(GS_ERR_INVALID_ARG, "PLY layout is NULL");
    if (L->stride < 4 || L->stride > kPlyMaxStride) return ply_fail("PLY vertex stride out of range 4..1024");
    if (!(L->sh_rest == 0 || L->sh_rest == 3 || L->sh_rest == 8 || L->sh_rest == 15))
        return ply_fail("PLY f_rest coefficients per channel must be 0, 3, 8 or 15");
    auto ok = [&](int32_t off) { return off >= 0 && (uint32_t)off + 4u <= L->stride; };
    for (int k = 0; k < 3; ++k)
        if (!ok(L->pos[k]) || !ok(L->f_dc[k]) || !ok(L->scale[k])) return ply_fail("PLY field offset outside a vertex");
    for (int k = 0; k < 4; ++k)
        if (!ok(L->rot[k])) return ply_fail("PLY field offset outside a vertex");
    if (!ok(L->opacity)) return ply_fail("PLY field offset outside a vertex");
    for (uint32_t k = 0; k < 3 * L->sh_rest; ++k)
        if (!ok(L->f_rest[k])) return ply_fail("PLY field offset outside a vertex");
    return GS_OK;
}

}  // namespace gs

using namespace gs;

extern "C" gs_status gs_ply_parse_header(const void *bytes, size_t len, gs_ply_layout *out) {
    if (!bytes || !out) return set_error(GS_ERR_INVALID_ARG, "NULL argument");
    const char *p = static_cast<const char *>(bytes);
    static const char kEnd[] = "end_header\n";
    const size_t kEndLen = sizeof(kEnd) - 1;
    if (len < 3 || std::memcmp(p, "ply", 3) != 0) return ply_fail("not a PLY file");
    size_t end = std::string::npos;
    for (size_t i = 0; i + kEndLen <= len; ++i) {
        if (p[i] == 'e' && std::memcmp(p + i, kEnd, kEndLen) == 0) {
            end = i;
            break;
        }
    }
    if (end == std::string::npos) return ply_fail("PLY header has no end_header line");
    const std::string head(p, end);

    gs_ply_layout L;
    std::memset(&L, 0, sizeof(L));
    int32_t *req[14] = {&L.pos[0], &L.pos[1], &L.pos[2], &L.f_dc[0], &L.f_dc[1], &L.f_dc[2], &L.opacity,
                        &L.scale[0], &L.scale[1], &L.scale[2], &L.rot[0], &L.rot[1], &L.rot[2], &L.rot[3]};
    static const char *kReq[14] = {"x", "y", "z", "f_dc_0", "f_dc_1", "f_dc_2", "opacity",
                                   "scale_0", "scale_1", "scale_2", "rot_0", "rot_1", "rot_2", "rot_3"};
    for (int k = 0; k < 14; ++k) *req[k] = -1;
    for (int k = 0; k < 45; ++k) L.f_rest[k] = -1;

    struct Element {
        std::string name;
        uint64_t count = 0, stride = 0;
        bool has_list = false;
    };
    std::vector<Element> elems;
    std::string format;
    uint32_t rest_seen = 0;
    size_t pos = 0;
    bool magic = true;
    while (pos < head.size()) {
        size_t nl = head.find('\n', pos);
        if (nl == std::string::npos) nl = head.size();
        const std::vector<std::string> t = split_ws(head.substr(pos, nl - pos));
        pos = nl + 1;
        if (magic) {  // the "ply" line
            magic = false;
            continue;
        }
        if (t.empty() || t[0] == "comment" || t[0] == "obj_info") continue;
        if (t[0] == "format") {
            if (t.size() < 2) return ply_fail("PLY format line is malformed");
            format = t[1];
        } else if (t[0] == "element") {
            Element e;
            if (t.size() < 3 || !parse_u64(t[2], &e.count)) return ply_fail("PLY element line is malformed");
            e.name = t[1];
            if (e.name == "vertex")
                for (const Element &o : elems)
                    if (o.name == "vertex") return ply_fail("PLY has two vertex elements");
            elems.push_back(e);
        } else if (t[0] == "property") {
            if (elems.empty()) return ply_fail("PLY property before any element");
            Element &e = elems.back();
            if (t.size() >= 2 && t[1] == "list") {
                if (e.name == "vertex") return ply_fail("list properties are not supported in the vertex element");
                e.has_list = true;
                continue;
            }
            if (t.size() < 3) return ply_fail("PLY property line is malformed");
            const int b = ply_type_bytes(t[1]);
            if (!b) return ply_fail("unknown PLY property type '%s'", t[1].c_str());
            if (e.name == "vertex") {
                const std::string &name = t[2];
                for (int k = 0; k < 14; ++k) {
                    if (name == kReq[k]) {
                        if (!is_float32(t[1])) return ply_fail("PLY property '%s' must be float", kReq[k]);
                        *req[k] = (int32_t)e.stride;
                    }
                }
                if (name.rfind("f_rest_", 0) == 0) {
                    uint64_t idx = 0;
                    if (!parse_u64(name.substr(7), &idx) || idx >= 45)
                        return ply_fail("PLY property '%s' is beyond SH degree 3", name.c_str());
                    if (!is_float32(t[1])) return ply_fail("PLY property '%s' must be float", name.c_str());
                    L.f_rest[idx] = (int32_t)e.stride;
                    ++rest_seen;
                }
                if (e.stride + (uint64_t)b > kPlyMaxStride) return ply_fail("PLY vertex stride out of range 4..1024");
            }
            e.stride += (uint64_t)b;
        } else {
            return ply_fail("unknown PLY header line '%s'", t[0].c_str());
        }
    }
    if (format != "binary_little_endian") return ply_fail("unsupported PLY format '%s'", format.c_str());
    // the vertex block follows the elements declared before it
    uint64_t before = 0, count = 0, vstride = 0;
    bool seen_vertex = false;
    for (const Element &e : elems) {
        if (e.name == "vertex") {
            seen_vertex = true;
            count = e.count;
            vstride = e.stride;
            break;
        }
        if (e.has_list) return ply_fail("PLY element '%s' before the vertex element has a list property", e.name.c_str());
        before += e.count * e.stride;
    }
    if (!seen_vertex) return ply_fail("PLY has no vertex element");
    if (count > 0xFFFFFFFFull) return ply_fail("PLY vertex count above 2^32 - 1");
    for (int k = 0; k < 14; ++k)
        if (*req[k] < 0) return ply_fail("PLY vertex element lacks property '%s'", kReq[k]);
    if (!(rest_seen == 0 || rest_seen == 9 || rest_seen == 24 || rest_seen == 45))
        return ply_fail("PLY f_rest count must be 0, 9, 24 or 45");
    for (uint32_t k = 0; k < rest_seen; ++k)
        if (L.f_rest[k] < 0) return ply_fail("PLY f_rest properties are not numbered 0..n-1");
    L.data_offset = (uint64_t)end + kEndLen + before;
    L.count = (uint32_t)count;
    L.stride = (uint32_t)vstride;
    L.sh_rest = rest_seen / 3;
    const gs_status s = ply_check_layout(&L);
    if (s != GS_OK) return s;
    *out = L;
    return GS_OK;
}

namespace gs {

struct PlyParams {
    gs_ply_layout L;
    const uint8_t *vertices;
    uint8_t *records;
    uint32_t wide;  // vertices 16-byte aligned: whole CTAs stage by 16-byte copies
};

__device__ __forceinline__ uint32_t f16_bits(float x) { return (uint32_t)__half_as_ushort(__float2half_rn(x)); }
__device__ __forceinline__ uint32_t bf16_bits(float x) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x));
}

// 2^(j/32), j = 0..31, as pairs of floats (exp_certain), copied to shared memory by each CTA.
__constant__ Two c_exp_table[GS_EXP_TABLE_SIZE] = GS_EXP_TABLE;

// A vertex's fields in the staged bytes.  ALIGNED: the vertex starts on a word, every field lies
// on a word, and f_rest is one ascending run, so a field is one shared load at a constant distance
// from a base; otherwise a field is one or two words joined by a funnel shift.
template <bool ALIGNED>
struct StagedVertex {
    const gs_ply_layout &L;
    const uint32_t *s;
    uint32_t base;  // byte of the vertex in the staged words

    __device__ __forceinline__ float at(int32_t off) const {
        const uint32_t b = base + (uint32_t)off, w = b >> 2;
        if constexpr (ALIGNED) return __uint_as_float(s[w]);
        const uint32_t sh = (b & 3u) * 8u;
        uint32_t v = s[w];
        if (sh) v = __funnelshift_r(v, s[w + 1], sh);
        return __uint_as_float(v);
    }

    // SH coefficient k of channel c: f_rest is channel-major (K coefficients of R, then G, then B)
    __device__ __forceinline__ float sh(uint32_t K, uint32_t k, uint32_t c) const {
        if (k >= K) return 0.0f;
        if constexpr (ALIGNED) return __uint_as_float(s[((base + (uint32_t)L.f_rest[0]) >> 2) + c * K + k]);
        return at(L.f_rest[c * K + k]);
    }
};

// The double path of the colour (rgb = 0.5 + SH_C0·f_dc and a = sigmoid(opacity), to 8 bits), of
// a scale and of a rotation: taken where the float path is not certain of its rounding.
__device__ __noinline__ uint32_t ply_unorm8_dc(float dc) { return unorm8_rne(0.5 + kShC0 * (double)dc); }
__device__ __noinline__ uint32_t ply_unorm8_opacity(float op) { return unorm8_rne(1.0 / (1.0 + exp(-(double)op))); }
__device__ __noinline__ float ply_scale(float s) { return (float)exp((double)s); }
__device__ __noinline__ float4 ply_rot(float x, float y, float z, float w) {
    const double q[4] = {x, y, z, w};
    const double nrm = sqrt(((q[0] * q[0] + q[1] * q[1]) + q[2] * q[2]) + q[3] * q[3]);
    return make_float4((float)(q[0] / nrm), (float)(q[1] / nrm), (float)(q[2] / nrm), (float)(q[3] / nrm));
}
struct Cov3d {
    float v[6];
};
__device__ __noinline__ Cov3d ply_cov3d(float4 r, float s0, float s1, float s2) {
    const float rot[4] = {r.x, r.y, r.z, r.w}, scale[3] = {s0, s1, s2};
    Cov3d c;
    cov3d_from_rot_scale(rot, scale, c.v);
    return c;
}

// Half records leave through rows padded to 144 bytes (dense 128-byte rows would put a
// quarter-warp's 16-byte stores on one bank).
template <uint32_t FMT>
constexpr uint32_t kPlyRowBytes = (FMT == GS_FORMAT_FP32) ? 224u : 144u;

// Tiles ahead of its own whose vertex bytes a CTA asks L2 for (as the preprocess does).
constexpr uint32_t kPlyPrefetchTiles = 152 * 4;

template <uint32_t FMT, bool ALIGNED>
__global__ void __launch_bounds__(kPlyThreads) ply_convert_kernel(const __grid_constant__ PlyParams P) {
    constexpr uint32_t REC = (FMT == GS_FORMAT_FP32) ? 224u : 128u;
    constexpr uint32_t ROW16 = kPlyRowBytes<FMT> / 16;
    // The staged vertex words, and after all threads hold their records in registers, the rows of
    // the records in the same bytes: half the shared memory, so more CTAs an SM.
    extern __shared__ __align__(16) uint8_t smem[];
    uint32_t *s_in = reinterpret_cast<uint32_t *>(smem);
    uint4 *s_out = reinterpret_cast<uint4 *>(smem);
    __shared__ Two s_table[GS_EXP_TABLE_SIZE];
    const gs_ply_layout &L = P.L;
    const uint32_t tid = threadIdx.x;
    const uint64_t first = (uint64_t)blockIdx.x * kPlyThreads;
    const uint32_t cnt = (uint32_t)min((uint64_t)kPlyThreads, (uint64_t)L.count - first);
    const bool wide = P.wide && cnt == kPlyThreads;  // 128 × stride bytes from a 16-byte boundary
    if (tid < GS_EXP_TABLE_SIZE) s_table[tid] = c_exp_table[tid];

    // ---- stage the CTA's vertex bytes [b0, b1) ----
    const uint64_t b0 = first * L.stride, b1 = (first + cnt) * L.stride;
    const uint64_t w0 = b0 >> 2;
    if (wide) {
        const uint4 *src = reinterpret_cast<const uint4 *>(P.vertices + b0);
        const uint32_t chunks = kPlyThreads * L.stride / 16u;
        for (uint32_t q = tid; q < chunks; q += kPlyThreads) cp_async16(smem + 16u * q, src + q);
        const uint64_t ahead = first + (uint64_t)kPlyPrefetchTiles * kPlyThreads;
        if (tid == 0 && ahead + kPlyThreads <= L.count)
            prefetch_l2_bulk(P.vertices + ahead * L.stride, kPlyThreads * L.stride);
        cp_async_wait_all();
    } else {
        // the words that cover the bytes; a block's last, partial word is read bytewise
        const uint64_t total = (uint64_t)L.count * L.stride, w1 = (b1 + 3) >> 2, whole = total >> 2;
        const uint32_t nw = (uint32_t)(w1 - w0);
        const uint32_t *v32 = reinterpret_cast<const uint32_t *>(P.vertices);
        for (uint32_t k = tid; k < nw; k += kPlyThreads) {
            const uint64_t w = w0 + k;
            uint32_t v;
            if (w < whole) {
                v = __ldcs(v32 + w);
            } else {
                v = 0;
                for (uint32_t j = 0; j < 4; ++j)
                    if (w * 4 + j < total) v |= (uint32_t)P.vertices[w * 4 + j] << (8 * j);
            }
            s_in[k] = v;
        }
    }
    __syncthreads();

    uint32_t rec[REC / 4];  // the record, in words
    if (tid < cnt) {
        const StagedVertex<ALIGNED> V{L, s_in, (uint32_t)((first + tid) * L.stride - (w0 << 2))};
        // colour: floats within 1e-4 of 255·channel settle all but the halfway cases
        uint32_t color = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float dc = V.at(L.f_dc[c]);
            uint32_t u;
            if (!unorm8_certain(fmaf(dc, (float)(255.0 * kShC0), 127.5f), 1e-4f, &u)) u = ply_unorm8_dc(dc);
            color |= u << (8 * c);
        }
        {
            const float op = V.at(L.opacity);
            uint32_t u;
            if (!unorm8_certain(255.0f / (1.0f + expf(-op)), 1e-4f, &u)) u = ply_unorm8_opacity(op);
            color |= u << 24;
        }
        float scale[3], rot[4];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float s = V.at(L.scale[k]);
            if (!exp_certain(s, s_table, &scale[k])) scale[k] = ply_scale(s);
        }
        {
            const float q[4] = {V.at(L.rot[1]), V.at(L.rot[2]), V.at(L.rot[3]), V.at(L.rot[0])};  // x, y, z, w
            if (!unit_quat_certain(q, [](float s) { return rsqrtf(s); }, rot)) {
                const float4 r = ply_rot(q[0], q[1], q[2], q[3]);
                rot[0] = r.x;
                rot[1] = r.y;
                rot[2] = r.z;
                rot[3] = r.w;
            }
        }
        const uint32_t K = L.sh_rest;
#pragma unroll
        for (int k = 0; k < 3; ++k) rec[k] = __float_as_uint(V.at(L.pos[k]));
        rec[3] = color;
        if constexpr (FMT == GS_FORMAT_FP32) {
            float cov[6];
            if (!cov3d_certain(rot, scale, cov)) {
                const Cov3d c = ply_cov3d(make_float4(rot[0], rot[1], rot[2], rot[3]), scale[0], scale[1], scale[2]);
#pragma unroll
                for (int k = 0; k < 6; ++k) cov[k] = c.v[k];
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) rec[49 + k] = __float_as_uint(cov[k]);
            rec[55] = 0u;
#pragma unroll
            for (int k = 0; k < 15; ++k)
#pragma unroll
                for (int c = 0; c < 3; ++c) rec[4 + 3 * k + c] = __float_as_uint(V.sh(K, k, c));
        } else {
            // 16-bit units from byte 16: rot, scale, SH, padding
            rec[4] = f16_bits(rot[0]) | (f16_bits(rot[1]) << 16);
            rec[5] = f16_bits(rot[2]) | (f16_bits(rot[3]) << 16);
            rec[6] = f16_bits(scale[0]) | (f16_bits(scale[1]) << 16);
            rec[7] = f16_bits(scale[2]);
            auto sh16 = [&](int i) {  // unit i of the SH run
                const float v = V.sh(K, i / 3, i % 3);
                return (FMT == GS_FORMAT_HALF_SH_FP16) ? f16_bits(v) : bf16_bits(v);
            };
            rec[7] |= sh16(0) << 16;
#pragma unroll
            for (int i = 1; i < 45; i += 2) rec[8 + i / 2] = sh16(i) | (sh16(i + 1) << 16);
            rec[30] = rec[31] = 0u;
        }
    }
    __syncthreads();  // every vertex is in registers: the rows may take its place
    if (tid < cnt) {
        uint4 *row = s_out + tid * ROW16;
#pragma unroll
        for (uint32_t k = 0; k < REC / 16; ++k)
            row[k] = make_uint4(rec[4 * k], rec[4 * k + 1], rec[4 * k + 2], rec[4 * k + 3]);
    }
    uint8_t *dst = P.records + first * REC;
    if constexpr (FMT == GS_FORMAT_FP32) {
        // one bulk store of the CTA's records (generic-proxy writes made visible to it first)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            const uint32_t src = (uint32_t)__cvta_generic_to_shared(s_out);
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src),
                         "r"(cnt * REC)
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else {
        __syncthreads();
        constexpr uint32_t C16 = REC / 16;
        uint4 *d16 = reinterpret_cast<uint4 *>(dst);
        for (uint32_t q = tid; q < cnt * C16; q += kPlyThreads) d16[q] = s_out[(q / C16) * ROW16 + q % C16];
    }
}

// Whether every field of a vertex lies on a word and f_rest is one ascending run of floats.
static bool ply_layout_aligned(const gs_ply_layout &L) {
    uint32_t low = L.stride;
    for (int k = 0; k < 3; ++k) low |= (uint32_t)(L.pos[k] | L.f_dc[k] | L.scale[k]);
    for (int k = 0; k < 4; ++k) low |= (uint32_t)L.rot[k];
    low |= (uint32_t)L.opacity;
    for (uint32_t k = 0; k < 3 * L.sh_rest; ++k) {
        low |= (uint32_t)L.f_rest[k];
        if (L.f_rest[k] != L.f_rest[0] + 4 * (int32_t)k) return false;
    }
    return (low & 3u) == 0;
}

template <uint32_t FMT, bool ALIGNED>
cudaError_t launch_ply_fmt(const PlyParams &P, cudaStream_t st) {
    auto smem_of = [](uint32_t stride) {
        const size_t in = align_up((size_t)kPlyThreads * stride + 8, 16), out = kPlyThreads * kPlyRowBytes<FMT>;
        return in > out ? in : out;
    };
    cudaError_t e = cudaFuncSetAttribute(ply_convert_kernel<FMT, ALIGNED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem_of(kPlyMaxStride));
    if (e != cudaSuccess) return e;
    const uint32_t grid = (P.L.count + kPlyThreads - 1) / kPlyThreads;
    ply_convert_kernel<FMT, ALIGNED><<<grid, kPlyThreads, smem_of(P.L.stride), st>>>(P);
    count_launches(1);
    return cudaGetLastError();
}

template <uint32_t FMT>
cudaError_t launch_ply_layout(const PlyParams &P, cudaStream_t st) {
    return ply_layout_aligned(P.L) ? launch_ply_fmt<FMT, true>(P, st) : launch_ply_fmt<FMT, false>(P, st);
}

cudaError_t launch_ply_convert(const void *vertices, const gs_ply_layout &L, uint32_t format, void *records,
                               cudaStream_t st) {
    if (L.count == 0) return cudaSuccess;
    PlyParams P;
    P.L = L;
    P.vertices = static_cast<const uint8_t *>(vertices);
    P.records = static_cast<uint8_t *>(records);
    P.wide = (uintptr_t)vertices % 16 == 0 ? 1u : 0u;
    switch (format) {
        case GS_FORMAT_FP32:
            return launch_ply_layout<GS_FORMAT_FP32>(P, st);
        case GS_FORMAT_HALF_SH_FP16:
            return launch_ply_layout<GS_FORMAT_HALF_SH_FP16>(P, st);
        default:
            return launch_ply_layout<GS_FORMAT_HALF_SH_BF16>(P, st);
    }
}

}  // namespace gs

extern "C" gs_status gs_ply_convert(const void *vertices, const gs_ply_layout *layout, uint32_t format,
                                    void *records, gs_stream stream) {
    const gs_status s = ply_check_layout(layout);
    if (s != GS_OK) return s;
    if (!(format == GS_FORMAT_FP32 || format == GS_FORMAT_HALF_SH_FP16 || format == GS_FORMAT_HALF_SH_BF16))
        return set_error(GS_ERR_INVALID_ARG, "unknown record format");
    if (layout->count == 0) return GS_OK;
    if (!vertices || !records) return set_error(GS_ERR_INVALID_ARG, "NULL argument");
    if ((uintptr_t)vertices % 4 != 0) return set_error(GS_ERR_INVALID_ARG, "vertices must be 4-byte aligned");
    if ((uintptr_t)records % 16 != 0) return set_error(GS_ERR_INVALID_ARG, "records must be 16-byte aligned");
    const cudaError_t e = launch_ply_convert(vertices, *layout, format, records, stream);
    if (e != cudaSuccess) return set_error(GS_ERR_CUDA, cudaGetErrorString(e));
    return GS_OK;
}
