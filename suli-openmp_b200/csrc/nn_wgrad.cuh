// nn_wgrad.cuh — weight gradient of a 3x3x3 convolution on the tensor cores (mma.sync m16n8k16,
// BF16 x BF16 -> FP32): dW[tap][co][ci] = sum_v dZ[v][co] X[v + off(tap)][ci], db[co] = sum_v dZ[v][co].
//
// The contraction runs over the voxels, so one staged block of dZ and of X serves all 27 taps:
// a CTA owns a column of 16 x 8 voxels and marches it up a segment of z-planes, with the planes
// of X (and its halo of one voxel) in a ring of four shared-memory slots and those of dZ in two,
// filled by cp.async one plane ahead.  Each of its nine warps owns one (dy, dz) pair: per row of 16
// voxels it loads the A fragments (16 MB output channels, voxels along K) once and, for its three
// dx, the B fragments of the row shifted by dx (voxels along K, 16 NB input channels), and keeps
// all 3 x 2 MB NB accumulator tiles in registers, so no partial sums are exchanged.  Rows are padded
// by 16 bytes, which makes the eight row addresses of an ldmatrix phase hit distinct banks.
//
// Measured at 128^3 (in brackets one tap a CTA, which stages both operands 27 times): 16 -> 16 channels
// 150 us (1709), 48 -> 16 344 (3033), 96 -> 32 at 64^3 240 (800); a gradient of the whole network 4.9
// ms (14.7).  No unit is full: the tensor pipe is busy 41-52 % of the time, L1 with the ldmatrix reads
// 38-63 %; the warps wait for fixed latencies and at the plane's barrier (27 instead of 18 warps an SM
// change nothing).
// Why mma.sync: 16-channel layers have a 16 x 16 output a tap, far below tcgen05's 64-row minimum,
// and the taps' shifted operands have no uniform stride that would stack them into its rows.
//
// Each CTA writes its sums to its own row of part (27 COUT CIN weights, then COUT biases; the CTAs
// of a row's channel blocks write disjoint parts) and k_sum_parts adds the rows in a fixed order.
#pragma once

namespace suli {
namespace nn {

constexpr int kWgX = 16, kWgY = 8;                        // voxels of a column's plane
constexpr int kWgHX = kWgX + 2, kWgHY = kWgY + 2;          // with the halo
constexpr int kWgThreads = 288;
constexpr int kWgSlotsX = 4, kWgSlotsZ = 2;
template <int MB, int NB>
struct WgGeo {
    static constexpr int RX = 32 * NB + 16, RZ = 32 * MB + 16;             // row pitches (bytes)
    static constexpr int XB = kWgHX * kWgHY * RX, ZB = kWgX * kWgY * RZ;   // a plane's bytes
    static constexpr int ACC = 24 * MB * NB;                                // accumulators a thread
    // The tensor cores' FP32 accumulation truncates, so a chain of n products is off by about
    // n/2 2^-24 of its sum: after CHAIN planes (8 products a plane) the accumulators are added, in
    // rounded FP32, to totals in shared memory (few channels), or a segment holds no more planes
    static constexpr bool TOTALS = MB * NB <= 2;
    static constexpr int CHAIN = MB * NB == 1 ? 8 : (MB * NB == 2 ? 16 : 32);
    static constexpr int RING = kWgSlotsX * XB + kWgSlotsZ * ZB;
    static constexpr int SMEM = RING + (TOTALS ? ACC * kWgThreads * 4 : 0);
    static constexpr int CTAS = MB * NB == 1 ? 3 : (MB * NB <= 3 ? 2 : 1);   // an SM holds at least
};

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                                  uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
// 16 bytes to shared memory, or zeros
__device__ __forceinline__ void wg_copy16(uint32_t dst, const void* src, bool valid) {
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ float wg_pair(uint32_t a) {   // sum of a register's two BF16 values
    return __uint_as_float(a << 16) + __uint_as_float(a & 0xffff0000u);
}

// grid: (columns x segments, channel blocks); seg = planes of a segment
template <int MB, int NB>
__global__ void __launch_bounds__(kWgThreads, (WgGeo<MB, NB>::CTAS)) k_wgrad_tc(Vol vol, ConvIn in, int cout, const __nv_bfloat16* __restrict__ dz,
                                                        int seg, float* part) {
    using Geo = WgGeo<MB, NB>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float sb[9][16 * MB];
    const uint32_t xs = smem_u32(smem), zs = xs + kWgSlotsX * Geo::XB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cin = in.ca + in.cb, ciblocks = cin / (16 * NB);
    const int co0 = (blockIdx.y / ciblocks) * 16 * MB, ci0 = (blockIdx.y % ciblocks) * 16 * NB;
    const int tx = (vol.nx + kWgX - 1) / kWgX, ty = (vol.ny + kWgY - 1) / kWgY;
    const int x0 = (blockIdx.x % tx) * kWgX, y0 = (blockIdx.x / tx % ty) * kWgY;
    const int z0 = (blockIdx.x / (tx * ty)) * seg, z1 = min(z0 + seg, vol.nz);
    const int hxn = (vol.nx + 1) / 2, hyn = (vol.ny + 1) / 2;

    auto stage_x = [&](int z) {   // plane z of X into its slot, zeros outside the volume
        const uint32_t slot = xs + ((z + kWgSlotsX) % kWgSlotsX) * Geo::XB;
        for (int q = tid; q < kWgHX * kWgHY * 2 * NB; q += kWgThreads) {
            const int v = q / (2 * NB), ch = (q % (2 * NB)) * 8;
            const int x = x0 + v % kWgHX - 1, y = y0 + v / kWgHX - 1, c = ci0 + ch;
            const bool ok = x >= 0 && x < vol.nx && y >= 0 && y < vol.ny && z >= 0 && z < vol.nz;
            const __nv_bfloat16* src = dz;
            if (ok) {
                const long long vi = (long long)x + vol.nx * ((long long)y + (long long)vol.ny * z);
                if (c >= in.ca) src = in.b + vi * in.cb + (c - in.ca);
                else if (in.a_half) src = in.a + ((long long)(x >> 1) + hxn * ((long long)(y >> 1) + (long long)hyn * (z >> 1))) * in.ca + c;
                else src = in.a + vi * in.ca + c;
            }
            wg_copy16(slot + v * Geo::RX + ch * 2, src, ok);
        }
    };
    auto stage_z = [&](int z) {   // plane z of dZ
        const uint32_t slot = zs + (z % kWgSlotsZ) * Geo::ZB;
        for (int q = tid; q < kWgX * kWgY * 2 * MB; q += kWgThreads) {
            const int v = q / (2 * MB), ch = (q % (2 * MB)) * 8;
            const int x = x0 + v % kWgX, y = y0 + v / kWgX;
            const bool ok = x < vol.nx && y < vol.ny;
            const __nv_bfloat16* src =
                ok ? dz + ((long long)x + vol.nx * ((long long)y + (long long)vol.ny * z)) * cout + co0 + ch : dz;
            wg_copy16(slot + v * Geo::RZ + ch * 2, src, ok);
        }
    };

    float acc[MB][NB][3][2][4];
#pragma unroll
    for (int a = 0; a < MB; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[a][b][d][h][e] = 0.f;
    float bias[MB][2];
#pragma unroll
    for (int a = 0; a < MB; ++a) bias[a][0] = bias[a][1] = 0.f;

    float* tot = reinterpret_cast<float*>(smem + Geo::RING) + tid;   // this thread's totals, kWgThreads apart
    auto each = [&](auto f) {   // f(accumulator, its number)
        int i = 0;
#pragma unroll
        for (int a = 0; a < MB; ++a)
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int d = 0; d < 3; ++d)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 4; ++e) f(acc[a][b][d][h][e], i++);
    };
    if (Geo::TOTALS) each([&](float&, int i) { tot[i * kWgThreads] = 0.f; });

    stage_x(z0 - 1);
    stage_x(z0);
    stage_x(z0 + 1);
    stage_z(z0);
    const int wy = warp % 3, wz = warp / 3;   // this warp's dy + 1, dz + 1
    // A: lane -> matrix m = lane / 8 (channels 8 (m & 1), voxels 8 (m >> 1)), row lane % 8;
    // B: lanes 0-15 the voxels of channels 0-7, lanes 16-31 of channels 8-15
    const uint32_t aoff = ((lane & 7) + 8 * (lane >> 4)) * Geo::RZ + 16 * ((lane >> 3) & 1);
    const uint32_t boff = (lane & 15) * Geo::RX + 16 * (lane >> 4);
    for (int z = z0; z < z1; ++z) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();   // planes up to z + 1 of X and z of dZ are in; every warp is done with plane z - 1
        if (z + 1 < z1) {
            stage_x(z + 2);
            stage_z(z + 1);
        }
        const uint32_t zrow = zs + (z % kWgSlotsZ) * Geo::ZB + aoff;
        const uint32_t xrow = xs + ((z + wz - 1 + kWgSlotsX) % kWgSlotsX) * Geo::XB + wy * kWgHX * Geo::RX + boff;
#pragma unroll 2
        for (int y = 0; y < kWgY; ++y) {
            uint32_t A[MB][4];
#pragma unroll
            for (int a = 0; a < MB; ++a)
                ldmatrix_x4_trans(zrow + y * kWgX * Geo::RZ + 32 * a, A[a][0], A[a][1], A[a][2], A[a][3]);
            if ((z * kWgY + y) % 9 == warp)
#pragma unroll
                for (int a = 0; a < MB; ++a) {
                    bias[a][0] += wg_pair(A[a][0]) + wg_pair(A[a][2]);
                    bias[a][1] += wg_pair(A[a][1]) + wg_pair(A[a][3]);
                }
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4_trans(xrow + (y * kWgHX + d) * Geo::RX + 32 * b, b0, b1, b2, b3);
#pragma unroll
                    for (int a = 0; a < MB; ++a) {
                        mma_bf16(acc[a][b][d][0], A[a][0], A[a][1], A[a][2], A[a][3], b0, b1);
                        mma_bf16(acc[a][b][d][1], A[a][0], A[a][1], A[a][2], A[a][3], b2, b3);
                    }
                }
        }
        if (Geo::TOTALS && (z - z0) % Geo::CHAIN == Geo::CHAIN - 1)
            each([&](float& v, int i) {
                tot[i * kWgThreads] += v;
                v = 0.f;
            });
    }
    if (Geo::TOTALS) each([&](float& v, int i) { v += tot[i * kWgThreads]; });
    float* row = part + (long long)blockIdx.x * (27LL * cout * cin + cout);
#pragma unroll
    for (int a = 0; a < MB; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {   // accumulator rows lane / 4 (+ 8), columns 2 (lane % 4) + {0, 1}
                        const int co = co0 + 16 * a + (lane >> 2) + 8 * e, ci = ci0 + 16 * b + 8 * h + 2 * (lane & 3);
                        const int tap = d + 3 * wy + 9 * wz;
                        *reinterpret_cast<float2*>(row + ((long long)tap * cout + co) * cin + ci) =
                            make_float2(acc[a][b][d][h][2 * e], acc[a][b][d][h][2 * e + 1]);
                    }
    if (ci0 == 0) {
#pragma unroll
        for (int a = 0; a < MB; ++a)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float v = bias[a][e];
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if ((lane & 3) == 0) sb[warp][16 * a + (lane >> 2) + 8 * e] = v;
            }
        __syncthreads();
        if (tid < 16 * MB) {
            float v = 0.f;
            for (int w = 0; w < 9; ++w) v += sb[w][tid];
            row[27LL * cout * cin + co0 + tid] = v;
        }
    }
}

// out[q] += sum over the nparts rows of part[row][q]: eight threads a column take the rows in turn
// and their sums are added in thread order (a fixed order, so a gradient is the same from run to
// run).  Block (32, 8), one block a 32 columns.
__global__ void __launch_bounds__(256) k_sum_parts(int nparts, long long width, const float* __restrict__ part, float* out) {
    __shared__ float sh[8][32];
    const long long q = (long long)blockIdx.x * 32 + threadIdx.x;
    float s = 0.f;
    if (q < width)
#pragma unroll 8
        for (int r = threadIdx.y; r < nparts; r += 8) s += part[r * width + q];
    sh[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && q < width) {
        for (int w = 1; w < 8; ++w) s += sh[w][threadIdx.x];
        out[q] += s;
    }
}

}  // namespace nn
}  // namespace suli
