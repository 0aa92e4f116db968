// Light buffer construction for the brute-force sphere tables (wavefront.h
// LightBufferView), after Haines and Greenberg's light buffer (1986): around
// each point light a cube of direction cells, and per cell the spheres a
// shadow ray towards the light can meet when its origin, seen from the light,
// lies in that cell.  Built once per scene.
//
// Exactness.  A shadow ray (origin o = p + 1e-4 N on a sphere, direction
// L = normalize(light - p), occluded when some sphere has t > 0 and
// t^2 < |light - p|^2, Renderer.cu:348-352) runs the float test of
// trace.cuh.  A sphere that test accepts is passed by the exact ray within
// r + 4 sqrt(eps) D of its centre, D = |o - c| (the bound the LBVH walk uses,
// bvh_traverse.cuh), at a parameter between -4.5 sqrt(eps) D and the light.
// The ray stays within 2e-4 + kK |o - light| of the segment from the light to
// o (the 1e-4 offset and the float error of L), so that segment passes within
// R' = r + m + 2e-4 + kK dcap of the centre, m = kK (D + 1e-3) and
// D <= |c - light| + dcap, where dcap bounds |o - light| (every origin lies on
// a sphere; the lookup checks it).  Every point of the segment lies, seen from
// the light, in the origin's direction; so the sphere's cap of directions
// (half-angle asin(R' / |c - light|)) contains that direction, and the cell
// the lookup finds lists the sphere: a cell lists every sphere whose cap,
// widened by 1e-4 rad for the lookup's rounding, meets the cell's bounding
// cone.  A sphere whose centre lies within R' + m of the light (the segment
// could end inside it) is listed in every cell.  Spheres whose caps miss the
// bounding cone of the cell's whole face, widened by 8e-3 rad, are left out
// beforehand: the directions of a cell lie in that cone, so a cap that holds
// one of them, give or take the lookup's 1e-4 rad, meets it (a cap that meets
// only the part of a cell's bounding cone that sticks out of the face holds
// none).  The direction buffer's lists are built the same way (its own note
// below).
#include "light_buffer.h"

namespace atx {
namespace {

constexpr double kK = 1.2207031e-3;   // 5 sqrt(2^-24) per unit of distance, as kBvhK

uint64_t up(uint64_t x) { return (x + 255u) & ~uint64_t(255u); }

// A tile: the 4 x 8 cells of a cube face that one warp builds together, one
// cell per lane.  Its 8 cells along the second axis are neighbouring lines.
constexpr uint32_t kTileI = 4, kTileJ = 8;
__host__ __device__ constexpr uint32_t tiles_j(uint32_t res) { return (res + kTileJ - 1) / kTileJ; }
__host__ __device__ constexpr uint32_t tiles_for(uint32_t res)   // per face
{
    return ((res + kTileI - 1) / kTileI) * tiles_j(res);
}

// Scratch for the cell and tile cones (k_cells_prep) at the end of both buffers.
uint64_t cone_bytes(uint32_t res)
{
    const uint64_t tiles = 6u * tiles_for(res);
    return up(cells_for(res) * sizeof(float4)) + up(cells_for(res) * sizeof(float)) + up(tiles * sizeof(float4)) +
           up(tiles * sizeof(float));
}

struct Cones {
    float4* cell;      // axis, cosine of the half-angle
    float* cell_sin;
    float4* tile;
    float* tile_sin;
};

Cones carve_cones(unsigned char* p, uint32_t res)
{
    const uint64_t tiles = 6u * tiles_for(res);
    Cones c;
    c.cell = reinterpret_cast<float4*>(p);
    p += up(cells_for(res) * sizeof(float4));
    c.cell_sin = reinterpret_cast<float*>(p);
    p += up(cells_for(res) * sizeof(float));
    c.tile = reinterpret_cast<float4*>(p);
    p += up(tiles * sizeof(float4));
    c.tile_sin = reinterpret_cast<float*>(p);
    return c;
}

// Unit direction of face f (0..5: +x, -x, +y, -y, +z, -z) at in-face
// coordinates (u, v): the axes trace.cuh lb_cell divides by the face axis
// (face x: y, z; face y: x, z; face z: x, y).
__device__ float3 face_dir(uint32_t f, float u, float v)
{
    const uint32_t ax = f >> 1;
    float c[3];
    const uint32_t a = ax == 0 ? 1u : 0u, b = ax == 2 ? 1u : 2u;
    c[ax] = (f & 1u) ? -1.0f : 1.0f;
    c[a] = u;
    c[b] = v;
    const float s = 1.0f / sqrtf(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
    return make_float3(c[0] * s, c[1] * s, c[2] * s);
}

__device__ float dotf3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// Maximum of f(k) over k < n for a block of 256 threads, on thread 0.
template <class F>
__device__ float block_max(uint32_t n, F&& f)
{
    __shared__ float red[256];
    float mx = 0.0f;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) mx = fmaxf(mx, f(k));
    red[threadIdx.x] = mx;
    __syncthreads();
    for (uint32_t h = blockDim.x / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + h]);
        __syncthreads();
    }
    return red[0];
}

// Everything the cell lists need beforehand, in one launch of 256-thread
// blocks (each part is a few microseconds of latency, and a scene upload waits
// for all of them): cone_blocks blocks for the cones, one per light for its
// dcap, and the last one, when a direction buffer is built, for the reaches.
//
// Cones: one warp per tile, one cell per lane.  A cell's bounding cone is
// widened by 2e-4 rad (1e-4 for the lookup's rounding, the rest for the
// build's arithmetic): axis and the cosine of the half-angle in cell[], its
// sine in cell_sin[]; the farthest points of a cell from its centre are its
// corners.  A tile's cone holds its cells' cones and 8e-3 rad more: the cell
// test's slack of 2e-5 on a cosine is at most sqrt(4e-5) = 6.4e-3 rad, so a
// sphere that passes a cell's test passes its tile's.
//
// dcap[l] = max over spheres of |c - light| + r, plus 1: every shadow-ray
// origin (a hit point lifted by 1e-4) lies within it.
//
// reach_i: the sphere's radius, its 1e-4 surface offset and a float hit
// point's typical error (a hit point farther off falls back to the whole
// table), from E = max over spheres of |c|_1 + r, a bound on the coordinates
// the hit-point arithmetic sees.
__global__ void __launch_bounds__(256) k_cells_prep(const float4* __restrict__ sph, const float* __restrict__ rad,
                                                    uint32_t n, const DevLight* __restrict__ lights, uint32_t nl,
                                                    uint32_t res, uint32_t cone_blocks, Cones out, float* dcap,
                                                    float* reach)
{
    if (blockIdx.x < cone_blocks) {
        const uint32_t id = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
        const uint32_t T = tiles_for(res);
        if (id >= 6u * T) return;   // whole warps
        const uint32_t f = id / T, i0 = (id % T) / tiles_j(res) * kTileI, j0 = (id % T) % tiles_j(res) * kTileJ;
        const uint32_t i = i0 + lane / kTileJ, j = j0 + lane % kTileJ;
        const float fr = (float)res;
        const float3 axis = face_dir(f, (float)(2u * i0 + kTileI) / fr - 1.0f, (float)(2u * j0 + kTileJ) / fr - 1.0f);
        float wide = 0.0f;
        if (i < res && j < res) {
            const float u0 = 2.0f * i / fr - 1.0f, u1 = 2.0f * (i + 1) / fr - 1.0f;
            const float v0 = 2.0f * j / fr - 1.0f, v1 = 2.0f * (j + 1) / fr - 1.0f;
            const float3 ctr = face_dir(f, 0.5f * (u0 + u1), 0.5f * (v0 + v1));
            float cmin = 1.0f;
            for (int k = 0; k < 4; ++k)
                cmin = fminf(cmin, dotf3(ctr, face_dir(f, (k & 1) ? u1 : u0, (k & 2) ? v1 : v0)));
            const float hw = acosf(fminf(1.0f, cmin)) + 2e-4f;
            const uint32_t cell = (f * res + i) * res + j;
            out.cell[cell] = make_float4(ctr.x, ctr.y, ctr.z, cosf(hw));
            out.cell_sin[cell] = sinf(hw);
            wide = acosf(fminf(1.0f, dotf3(axis, ctr))) + hw;
        }
        for (int off = 16; off > 0; off >>= 1) wide = fmaxf(wide, __shfl_xor_sync(0xffffffffu, wide, off));
        if (lane == 0) {
            out.tile[id] = make_float4(axis.x, axis.y, axis.z, cosf(wide + 8e-3f));
            out.tile_sin[id] = sinf(wide + 8e-3f);
        }
    } else if (blockIdx.x - cone_blocks < nl) {
        const uint32_t l = blockIdx.x - cone_blocks;
        const DevLight lt = lights[l];
        const float mx = block_max(n, [&](uint32_t k) {
            const float4 s = sph[k];
            const float3 v = make_float3(s.x - lt.pos[0], s.y - lt.pos[1], s.z - lt.pos[2]);
            return sqrtf(dotf3(v, v)) + rad[k];
        });
        if (threadIdx.x == 0) dcap[l] = mx * 1.0001f + 1.0f;
    } else {
        const float e = block_max(n, [&](uint32_t k) {
            const float4 s = sph[k];
            return fabsf(s.x) + fabsf(s.y) + fabsf(s.z) + rad[k];
        });
        for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) reach[k] = rad[k] * 1.001f + 2e-4f + (float)kK * e;
    }
}

// ---------------------------------------------------------- direction buffer
//
// Exactness.  An extension ray leaves the sphere its path last hit: origin
// o = p + 1e-4 N with p the float hit point, direction d.  The lookup uses the
// lists of that sphere i only when |o - c_i| <= reach_i (checked per ray;
// else the whole table), so o = c_i + e with |e| <= reach_i.  A sphere j the
// float test accepts has a ray point X = o + t d, t >= -4.5 sqrt(eps) D_j,
// within r_j + 4 sqrt(eps) D_j of c_j (D_j = |o - c_j| <= |c_j - c_i| +
// reach_i).  Then c_i + t d = X - e lies within R' = r_j + m + reach_i of c_j,
// m = kK (D_j + 1e-3): for t >= 0 the ball (c_j, R') meets the cone of
// directions of d's cell from apex c_i, and for t < 0 its centre lies within
// R' + m of c_i.  A cell lists every sphere passing one of those two tests
// (cell cone widened by 2e-4 rad, bounds rounded towards listing), sphere i
// itself included.

// A sphere as the cell tests of one origin see it: centre from the origin and
// its distance, sine and cosine of the half-angle of its inflated ball's cap
// of directions; sb = -1: listed in every cell (the origin's neighbourhood
// overlaps it).  Every bound rounded towards listing.
struct Cap {
    float3 v;
    float dist, sb, cb;
};

// reach: the origins' distance from the cells' apex o (dcap for a light, reach_i
// for a sphere); e1 + e2: the inflation beyond the radius and the float margin.
__device__ Cap make_cap(float3 o, float reach, float e1, float e2, float4 s, float r)
{
    Cap c;
    c.v = make_float3(s.x - o.x, s.y - o.y, s.z - o.z);
    c.dist = sqrtf(dotf3(c.v, c.v));
    const float m = (float)kK * (c.dist + reach + 1e-3f);
    const float rp = r * 1.00001f + m + e1 + e2;
    if (!(c.dist > (rp + m) * 1.0001f)) {
        c.sb = -1.0f;
        c.cb = 0.0f;
    } else {
        c.sb = fminf(1.0f, rp / c.dist * 1.0001f);
        c.cb = sqrtf(fmaxf(0.0f, 1.0f - c.sb * c.sb));
    }
    return c;
}

__device__ __forceinline__ Cap shfl_cap(const Cap& c, int from)
{
    Cap x;
    x.v.x = __shfl_sync(0xffffffffu, c.v.x, from);
    x.v.y = __shfl_sync(0xffffffffu, c.v.y, from);
    x.v.z = __shfl_sync(0xffffffffu, c.v.z, from);
    x.dist = __shfl_sync(0xffffffffu, c.dist, from);
    x.sb = __shfl_sync(0xffffffffu, c.sb, from);
    x.cb = __shfl_sync(0xffffffffu, c.cb, from);
    return x;
}

// Whether a cap meets the cone (axis, half-angle with cosine ch and sine sh):
// cos(angle between the axes) >= cos(half-angle + beta), with a 2e-5 slack.
__device__ __forceinline__ bool cap_meets(float3 axis, float ch, float sh, const Cap& c)
{
    return c.sb < 0.0f || dotf3(axis, c.v) >= c.dist * (ch * c.cb - sh * c.sb - 2e-5f);
}

constexpr uint32_t kFaceCap = 2048;   // caps a block keeps in shared memory
constexpr size_t kCapBytes = sizeof(float4) + sizeof(float2) + sizeof(uint16_t);

// The cell lists of both buffers: one block of 256 threads per (apex, cube
// face, share of the face's tiles), the apexes n_db spheres from db_first on,
// then the nl lights.
//
// First the block keeps the spheres whose caps meet the face's bounding cone
// (its corners lie acos(1/sqrt 3) from the face axis), in index order, with
// their caps worked out once (a square root, a division and a square root each).
// Then a warp takes a tile of 32 cells at a time, one cell per lane: its lanes
// test 32 of those caps against the tile's cone, and each cap that passes is
// handed to all lanes, which test it against their own cells and append it to
// their lists, staged in shared memory and written as whole 32-byte sectors.
// A cap is tested against a cell only when it meets the cell's tile, and that
// test is a dot product and a comparison.  One warp per cell testing every cap
// of the face (with its square roots and division) took 680 us for 256 spheres
// and 8 lights at 32 cells along an edge (1.6 M cells), this takes 47 us; 1,000
// spheres and 12 lights 5,430 -> 317 us.  Bound by issue; the sectors written
// are 50 MB for 256 spheres (8 us).  LINE: 16-bit words per cell line.
// More spheres than kFaceCap on a face: the tiles test all n (worked out on
// the fly).
template <uint32_t LINE>
__global__ void __launch_bounds__(256) k_cells_build(const float4* __restrict__ sph, const float* __restrict__ rad,
                                                     uint32_t n, uint32_t db_first, uint32_t n_db,
                                                     const float* __restrict__ reach,
                                                     uint16_t* db_line, const DevLight* __restrict__ lights,
                                                     const float* __restrict__ dcap, uint16_t* lb_line, uint32_t res,
                                                     uint32_t face_cap, Cones cones)
{
    constexpr uint32_t kRow = LINE / 2u + 1u;      // 32-bit words per staged line (odd: no bank conflicts)
    constexpr uint32_t kMax = LINE - 1u;           // spheres a line holds
    extern __shared__ float4 s_dyn[];              // face_cap x (v, dist), then (sb, cb), then the indices
    float4* f_v = s_dyn;
    float2* f_sc = reinterpret_cast<float2*>(f_v + face_cap);
    uint16_t* f_id = reinterpret_cast<uint16_t*>(f_sc + face_cap);
    __shared__ uint32_t stage[8][32 * kRow];
    __shared__ uint32_t warp_n[8];
    const uint32_t apex = blockIdx.x / 6u, f = blockIdx.x % 6u;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float3 o;
    float rho, e1, e2;
    uint16_t* line;
    if (apex < n_db) {
        const uint32_t i = db_first + apex;
        const float4 s = sph[i];
        o = make_float3(s.x, s.y, s.z);
        rho = reach[i];
        e1 = 0.0f, e2 = rho;
        line = db_line + (size_t)i * cells_for(res) * LINE;
    } else {
        const uint32_t l = apex - n_db;
        o = make_float3(lights[l].pos[0], lights[l].pos[1], lights[l].pos[2]);
        rho = dcap[l];
        e1 = 2e-4f, e2 = (float)kK * rho;
        line = lb_line + (size_t)l * cells_for(res) * LINE;
    }

    // the face's spheres, by an ordered compaction over the block
    const float3 axis = face_dir(f, 0.0f, 0.0f);
    const float hf = 0.95531662f + 8e-3f;   // acos(1/sqrt(3)), widened as a tile's cone
    const float chf = cosf(hf), shf = sinf(hf);
    uint32_t nc = 0;
    for (uint32_t base = 0; base < n; base += blockDim.x) {
        const uint32_t k = base + threadIdx.x;
        bool listed = false;
        Cap c;
        if (k < n) {
            c = make_cap(o, rho, e1, e2, sph[k], rad[k]);
            listed = cap_meets(axis, chf, shf, c);
        }
        const uint32_t mask = __ballot_sync(0xffffffffu, listed);
        if (lane == 0) warp_n[warp] = (uint32_t)__popc(mask);
        __syncthreads();
        uint32_t off = nc, tot = 0;
        for (uint32_t w = 0; w < 8u; ++w) {
            if (w < warp) off += warp_n[w];
            tot += warp_n[w];
        }
        const uint32_t at = off + __popc(mask & ((1u << lane) - 1u));
        if (listed && at < face_cap) {
            f_v[at] = make_float4(c.v.x, c.v.y, c.v.z, c.dist);
            f_sc[at] = make_float2(c.sb, c.cb);
            f_id[at] = (uint16_t)k;
        }
        nc += tot;
        __syncthreads();
    }
    const bool all = nc > face_cap;   // block-uniform
    if (all) nc = n;

    uint16_t* mine = reinterpret_cast<uint16_t*>(&stage[warp][lane * kRow]);
    const uint32_t T = tiles_for(res);
    for (uint32_t t = blockIdx.y * 8u + warp; t < T; t += gridDim.y * 8u) {
        const uint32_t i0 = t / tiles_j(res) * kTileI, j0 = t % tiles_j(res) * kTileJ;
        const uint32_t ci = i0 + lane / kTileJ, cj = j0 + lane % kTileJ;
        const bool me = ci < res && cj < res;
        const uint32_t cell = me ? (f * res + ci) * res + cj : f * res * res;
        const float4 cc = cones.cell[cell], tc = cones.tile[f * T + t];
        const float sh = cones.cell_sin[cell], tsh = cones.tile_sin[f * T + t];
        const float3 ctr = make_float3(cc.x, cc.y, cc.z), tax = make_float3(tc.x, tc.y, tc.z);
        uint32_t cnt = 0;
        for (uint32_t base = 0; base < nc; base += 32u) {
            const uint32_t q = base + lane;
            Cap c{};
            uint32_t id = q;
            bool pass = false;
            if (q < nc) {
                if (all) {
                    c = make_cap(o, rho, e1, e2, sph[q], rad[q]);
                } else {
                    const float4 a = f_v[q];
                    const float2 b = f_sc[q];
                    c = Cap{make_float3(a.x, a.y, a.z), a.w, b.x, b.y};
                    id = f_id[q];
                }
                pass = cap_meets(tax, tc.w, tsh, c);
            }
            uint32_t mask = __ballot_sync(0xffffffffu, pass);
            while (mask) {   // index order
                const int k = __ffs(mask) - 1;
                mask &= mask - 1u;
                const Cap x = shfl_cap(c, k);
                const uint32_t xi = __shfl_sync(0xffffffffu, id, k);
                if (cap_meets(ctr, cc.w, sh, x)) {
                    if (cnt < kMax) mine[1u + cnt] = (uint16_t)xi;
                    ++cnt;
                }
            }
        }
        mine[0] = (uint16_t)(cnt > kMax ? kLbAll : cnt);
        const uint32_t listed = me && cnt <= kMax ? cnt : 0u;
        uint32_t sectors = 1u;   // of 16 words, that the tile's longest list needs
        while (sectors < LINE / 16u && __any_sync(0xffffffffu, listed >= sectors * 16u)) ++sectors;
        __syncwarp();
        // eight lanes write 32 bytes of a cell: the count and 15 spheres, then 16
        // more where a list of the tile needs them
        for (uint32_t part = 0; part < sectors; ++part)
            for (uint32_t c0 = 0; c0 < 32u; c0 += 4u) {
                const uint32_t c = c0 + lane / 8u, w = part * 8u + lane % 8u;
                const uint32_t i = i0 + c / kTileJ, j = j0 + c % kTileJ;
                if (i < res && j < res)
                    reinterpret_cast<uint32_t*>(line + (size_t)((f * res + i) * res + j) * LINE)[w] =
                        stage[warp][c * kRow + w];
            }
        __syncwarp();
    }
}

}  // namespace

uint64_t lb_bytes(uint32_t nl, uint32_t res, uint32_t line_words)
{
    const uint64_t cells = (uint64_t)nl * cells_for(res);
    return up(cells * line_words * sizeof(uint16_t)) + up(nl * sizeof(float)) + cone_bytes(res) + 256;
}

uint64_t db_bytes(uint32_t n, uint32_t res, uint32_t line_words)
{
    const uint64_t cells = (uint64_t)n * cells_for(res);
    return up(cells * line_words * sizeof(uint16_t)) + up(n * sizeof(float)) + cone_bytes(res) + 256;
}

cudaError_t cells_build(const float4* sph, const float* radius, uint32_t n, const DevLight* lights, uint32_t nl,
                        uint32_t res, uint32_t line_words, void* lbuf, uint64_t lbytes, LightBufferView* lv,
                        void* dbuf, uint64_t dbytes, DirBufferView* dv, cudaStream_t stream, uint32_t db_first,
                        uint32_t db_count)
{
    const bool lb = lbuf != nullptr, db = dbuf != nullptr;
    if (!lb && !db) return cudaSuccess;
    if (n == 0 || n > kLbMaxSpheres || res < kCellResMin || res > kBvhLightRes ||
        (line_words != kLbLine && line_words != kBvhLine))
        return cudaErrorInvalidValue;
    if (lb && (nl == 0 || nl > kLbMaxLights || lbytes < lb_bytes(nl, res, line_words))) return cudaErrorInvalidValue;
    if (db && (n > kDbMaxBvhSpheres || dbytes < db_bytes(n, res, line_words) || db_first >= n))
        return cudaErrorInvalidValue;
    const uint64_t row = (uint64_t)cells_for(res) * line_words * sizeof(uint16_t);
    uint16_t* lline = static_cast<uint16_t*>(lbuf);
    uint16_t* dline = static_cast<uint16_t*>(dbuf);
    float *dcap = nullptr, *reach = nullptr;
    unsigned char* end = nullptr;   // the cones: in either buffer, both have the room
    if (lb) {
        dcap = reinterpret_cast<float*>(static_cast<unsigned char*>(lbuf) + up(nl * row));
        end = reinterpret_cast<unsigned char*>(dcap) + up(nl * sizeof(float));
    }
    if (db) {
        reach = reinterpret_cast<float*>(static_cast<unsigned char*>(dbuf) + up(n * row));
        end = reinterpret_cast<unsigned char*>(reach) + up(n * sizeof(float));
    }
    const Cones cones = carve_cones(end, res);
    const uint32_t apex_l = lb ? nl : 0u, apex_d = !db ? 0u : db_count < n - db_first ? db_count : n - db_first;
    if (apex_l + apex_d == 0u) return cudaErrorInvalidValue;
    const uint32_t cone_blocks = (6u * tiles_for(res) + 7u) / 8u;
    k_cells_prep<<<cone_blocks + apex_l + (db ? 1u : 0u), 256, 0, stream>>>(sph, radius, n, lights, apex_l, res,
                                                                           cone_blocks, cones, dcap, reach);
    const uint32_t cap = n < kFaceCap ? (n + 7u) & ~7u : kFaceCap;
    const size_t smem = cap * kCapBytes;
    // few apexes: a face's tiles over several blocks (each repeats the face's
    // compaction), about four blocks per SM of the GPU in all
    const uint32_t blocks = (apex_d + apex_l) * 6u, shares = (tiles_for(res) + 7u) / 8u;
    const uint32_t want = (600u + blocks - 1u) / blocks;
    const dim3 grid(blocks, want < shares ? want : shares);
    const auto build = line_words == kBvhLine ? k_cells_build<kBvhLine> : k_cells_build<kLbLine>;
    // the limit belongs to the function on this device, not to this call: always
    // the largest, so that a build on another thread never lowers it before this launch
    const cudaError_t e =
        cudaFuncSetAttribute(build, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kFaceCap * kCapBytes));
    if (e != cudaSuccess) return e;
    build<<<grid, 256, smem, stream>>>(sph, radius, n, db_first, apex_d, reach, dline, lights, dcap, lline, res, cap, cones);
    if (lb) *lv = LightBufferView{lline, dcap, nl, res};
    if (db) *dv = DirBufferView{dline, reach, n, res};
    return cudaGetLastError();
}

}  // namespace atx
