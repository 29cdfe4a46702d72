// fm_device.cuh -- small device helpers shared by the single-system kernels
// (fm_kernels.cu) and the multi-job slot engine (fm_engine.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fm_common.cuh"

namespace fm {

// |v|^2 in the reference's dot_product order, no contraction.
__device__ __forceinline__ double norm2_rn(double x, double y, double z)
{
    return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

// Programmatic dependent launch (kernels started with pdl_launch): wait for
// the predecessor grid to complete and its memory to be visible before
// touching anything, then let the successor grid begin launching.  Both are
// no-ops for a kernel launched without the attribute.
__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Set while a CUDA graph is being captured on this thread: its kernels are
// ordered by the graph's edges, launched without the attribute below.
extern thread_local bool pdl_capture;

// Launches k with programmatic stream serialization: the next kernel of the
// step may be launched while k's last blocks run, and waits in pdl_enter for
// k to complete before it reads anything (so the chain of small, often gated
// kernels of a step does not pay a full launch gap each).
template <typename... P, typename... A>
void pdl_launch(void (*k)(P...), dim3 grid, dim3 block, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = 0;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = pdl_capture ? 0 : 1;
    cudaLaunchKernelEx(&c, k, args...);
}

// pdl_launch with dynamic shared memory.
template <typename... P, typename... A>
void pdl_launch_smem(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = pdl_capture ? 0 : 1;
    cudaLaunchKernelEx(&c, k, args...);
}

// Neighbour-list entries are read once per step and never again before the
// next step: keep them out of L1, so that the partner positions they point at
// stay cached there.
__device__ __forceinline__ int4 ld_stream_int4(const int4 *p)
{
    int4 r;
    asm("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(p));
    return r;
}

__device__ __forceinline__ int2 ld_stream_int2(const int2 *p)
{
    int2 r;
    asm("ld.global.nc.L1::no_allocate.v2.s32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}

// Step s of lane `lane` of the TPM lanes that walk a row of cnt entries: four
// entries, of which number q counts while row_left > row_off(q). The lanes of a
// molecule take neighbouring entries, and slots ascend along a row, so a
// warp's gather of 32 partners meets fewer lines, of which L1 serves one a
// clock: by count over a 1M liquid's rows 21 with one lane a molecule and 13
// with four. row_first is the first entry of a step.
template <int TPM>
__device__ __forceinline__ int row_first(int s)
{
    return TPM == 1 ? 8 * (s >> 1) + 2 * (s & 1) : 4 * TPM * s;
}
template <int TPM>
__device__ __forceinline__ int row_left(int s, int lane, int cnt)
{
    return cnt - (TPM <= 2 ? row_first<TPM>(s) + 2 * lane : 4 * TPM * s + 8 * (lane >> 2) + (lane & 3));
}
template <int TPM>
__host__ __device__ constexpr int row_off(int q)
{
    return TPM <= 2 ? (q & 1) * 4 + (q >> 1) : (q >> 1) * 2 * TPM + (q & 1) * 4;
}
template <int TPM>
__device__ __forceinline__ int4 row_entries(const int32_t *L, int s, int lane, int left)
{
    if (TPM <= 2) {  // half a chunk: entries h, h + 4, h + 1, h + 5
        return ld_stream_int4(reinterpret_cast<const int4 *>(
            L + (TPM == 1 ? (size_t)(s >> 1) * 256u + 4 * (s & 1) : (size_t)s * 256u + 4 * lane)));
    }
    // entries t and t + 4 of two chunks
    const int32_t *p = L + (size_t)((TPM / 2) * s + (lane >> 2)) * 256u + 2 * (lane & 3);
    int2 a = make_int2(0, 0), b = make_int2(0, 0);
    if (left > 0) a = ld_stream_int2(reinterpret_cast<const int2 *>(p));
    if (left > row_off<TPM>(2)) b = ld_stream_int2(reinterpret_cast<const int2 *>(p + (TPM / 4) * 256));
    return make_int4(a.x, a.y, b.x, b.y);
}

// FP32 reciprocal of the precision form's pair magnitudes (s = 1/r^2): the
// hardware's approximate reciprocal (rcp.approx.ftz.f32, about 1 ulp; r^2 is
// never subnormal here), one instruction where a correctly rounded
// reciprocal takes a short sequence with a slow path.
__device__ __forceinline__ float rcp_f32(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Read-only gather of one double4 (32-byte aligned) as a single 256-bit load:
// one L1 request per partner instead of two.
__device__ __forceinline__ double4 ldg_pos(const double4 *p)
{
    double4 r;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
    return r;
}

// Sorts perm[b .. b+m) by key(perm value), by one lane (insertion).
template <typename K>
__device__ __forceinline__ void lane_sort_cell(int32_t *perm, int b, int m, K &&key_of)
{
    for (int x = b + 1; x < b + m; x++) {
        const int o = perm[x];
        const unsigned long long key = key_of(o);
        int y = x - 1;
        while (y >= b && key_of(perm[y]) > key) {
            perm[y + 1] = perm[y];
            y--;
        }
        perm[y + 1] = o;
    }
}

// Sorts perm[b .. b+m) by key(perm value), by one warp: up to 32 members by a
// bitonic sort in registers (as many stages as they need), up to 128 by rank,
// more by lane 0. Keys are distinct and below 2^59.
constexpr int SORT_RANK = 128;
template <typename K>
__device__ __forceinline__ void warp_sort_cell(int32_t *perm, int b, int m, int lane, K &&key_of)
{
    if (m <= 1) return;
    if (m <= 32) {
        unsigned long long key = ~0ull;
        int o = 0;
        if (lane < m) {
            o = perm[b + lane];
            key = key_of(o) << 5 | (unsigned)lane;
        }
        for (int k = 2; k < 2 * m; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, j);
                const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
                key = keep_min ? (key < other ? key : other) : (key > other ? key : other);
            }
        }
        o = __shfl_sync(0xffffffffu, o, (int)(key & 31u));
        if (lane < m) perm[b + lane] = o;
    } else if (m <= SORT_RANK) {
        unsigned long long key[SORT_RANK / 32];
        int o[SORT_RANK / 32], rank[SORT_RANK / 32];
#pragma unroll
        for (int q = 0; q < SORT_RANK / 32; q++) {
            const int x = q * 32 + lane;
            o[q] = x < m ? perm[b + x] : 0;
            key[q] = x < m ? key_of(o[q]) : ~0ull;
            rank[q] = 0;
        }
#pragma unroll
        for (int p = 0; p < SORT_RANK / 32; p++)
            for (int l = 0; l < 32; l++) {
                const unsigned long long other = __shfl_sync(0xffffffffu, key[p], l);
#pragma unroll
                for (int q = 0; q < SORT_RANK / 32; q++) rank[q] += other < key[q] ? 1 : 0;
            }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < SORT_RANK / 32; q++)
            if (q * 32 + lane < m) perm[b + rank[q]] = o[q];
    } else if (lane == 0) {
        lane_sort_cell(perm, b, m, key_of);
    }
}

// The same for four cells at once, each with eight lanes (lane & 7 of them,
// with its own b and m), where m <= 8; larger ones are left as they are.
template <typename K>
__device__ __forceinline__ void warp_sort_four_cells(int32_t *perm, int b, int m, int lane, K &&key_of)
{
    const int l8 = lane & 7;
    const bool mine = m <= 8 && l8 < m;
    unsigned long long key = ~0ull;
    int o = 0;
    if (mine) {
        o = perm[b + l8];
        key = (m > 1 ? key_of(o) : 0ull) << 3 | (unsigned)l8;
    }
#pragma unroll
    for (int k = 2; k <= 8; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, j);
            const bool keep_min = ((l8 & j) == 0) == ((l8 & k) == 0);
            key = keep_min ? (key < other ? key : other) : (key > other ? key : other);
        }
    }
    o = __shfl_sync(0xffffffffu, o, (lane & 24) | (int)(key & 7u));
    if (mine) perm[b + l8] = o;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Float min/max over the warp with one integer reduction each: the bit
// pattern with the magnitude bits flipped for negatives orders like the
// float (finite values).
__device__ __forceinline__ int float_order_key(float v)
{
    const int b = __float_as_int(v);
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float float_from_order_key(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }
__device__ __forceinline__ float warp_min(float v)
{
    return float_from_order_key(__reduce_min_sync(0xffffffffu, float_order_key(v)));
}
__device__ __forceinline__ float warp_max(float v)
{
    return float_from_order_key(__reduce_max_sync(0xffffffffu, float_order_key(v)));
}

// icell = ceiling((r + halfdomain)/cellsidelength) + 1 (1-based, halo = 1 and
// ncells+2); the 0-based extended index is the ceiling itself.  Out-of-grid
// values are clamped and flagged.
__device__ __forceinline__ int bin_axis(double x, double hd, double cs, int ne, bool &bad)
{
    double q = __ddiv_rn(__dadd_rn(x, hd), cs);
    if (!(q == q)) { bad = true; return 0; }
    int c = __double2int_ru(q);  // round toward +inf == ceiling for in-range values
    if (c < 0 || c > ne - 1) { bad = true; c = c < 0 ? 0 : ne - 1; }
    return c;
}

// Octant of extended cell (cx, cy, cz) that p lies in, x fastest. The
// line between two halves lies 2^-20 of a cell before their middle, so that a
// lattice site exactly in the middle falls in the same half whatever box of
// the periodic system its coordinate is rounded in.
__device__ __forceinline__ int sub_cell(const double4 &p, int cx, int cy, int cz, const double (&hd)[3],
                                        const double (&cs)[3])
{
    const float x = (float)((p.x + hd[0]) - (cx - 0.5) * cs[0]), y = (float)((p.y + hd[1]) - (cy - 0.5) * cs[1]);
    const float z = (float)((p.z + hd[2]) - (cz - 0.5) * cs[2]);
    const float tx = (float)cs[0] * -9.5367431640625e-7f, ty = (float)cs[1] * -9.5367431640625e-7f;
    const float tz = (float)cs[2] * -9.5367431640625e-7f;
    return (x > tx ? 1 : 0) | (y > ty ? 2 : 0) | (z > tz ? 4 : 0);
}

__device__ __forceinline__ bool is_halo(int x, int ne) { return x == 0 || x == ne - 1; }

// Periodic image of a coordinate: one FP64 add of +/-L, as the reference's
// halo copy r(k,np+m) = r(k,np+m) +/- domain(k).
__device__ __forceinline__ double image(double x, int s, double L)
{
    return s ? __dadd_rn(x, s > 0 ? L : -L) : x;
}

// Neumaier-compensated accumulation.
__device__ __forceinline__ void neumaier(double &sum, double &cmp, double x)
{
    double t = sum + x;
    cmp += fabs(sum) >= fabs(x) ? (sum - t) + x : (x - t) + sum;
    sum = t;
}

}  // namespace fm
