// Tiled form of the spatially variant image-space PSF (sm_100a).
//
// The kernel of a voxel is the LUT entry of its distance from the centre along
// each axis, so along x the LUT coordinate is constant over long segments.
// Each thread produces 8 consecutive x outputs of one row from a window held
// in registers: one shared-memory read per window element and one uniform
// 16-byte weight read per 4 taps serve 8 outputs, which leaves the products and
// sums themselves (two instructions per tap and output, rounded separately as
// the reference operator does) as the limit.  A block holds a tile of 32 x 32
// voxels of zt planes with its halo in shared memory (circular borders are
// resolved when the tile is filled); the lanes of a warp take 32 rows of one
// chunk of x, so a warp's LUT x coordinate is uniform.
//
// Forward: chunks end where the LUT x coordinate changes, so all 8 outputs use
// one kernel.  Adjoint: out[p] = sum_d in[p-d] w_{p-d}(d); the sources of a
// chunk may lie in several segments of each axis, and every combination of
// segments is added with its own kernel over its own sources.
//
// 192 x 192 x 96 voxels, 18 kernels of 5^3 to 9^3 taps: forward and adjoint 966
// + 4085 us with one voxel per thread reading through L1 (17 and 36
// instructions per tap), 382 + 672 us in this form, where instruction issue is
// 60 and 64 % active and the rows of a warp that lie in different segments of
// y (24 and 18 of 32 lanes active) are what is left.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace yrtb
{

// OperatorVarPsf (src/operators/OperatorVarPsf.cpp:290-455): every voxel has
// its own 3-D kernel, the LUT entry nearest to |voxel centre - image centre|
// (x, y, z gaps, clamped at the LUT's range).
struct VarPsfDev
{
	const float* w;     // all kernels' weights, z-major, then y, then x
	const int4* meta;   // per kernel: offset into w, half sizes x, y, z
	int lutX, lutY, lutZ;
	float gapX, gapY, gapZ;
	float vx, vy, vz;
	float cx, cy, cz;   // image centre: n * v / 2 in FP32
	int maxHx, maxHy, maxHz;
};

// LUT coordinate of index i along one axis (OperatorVarPsf::findNearestKernel
// with the distances of varconvolve: |(i + 0.5) v - centre| in FP64, then
// FP32, divided by the gap, rounded, clamped).  The LUT index of voxel
// (i, j, k) is a(i) + A (b(j) + B c(k)).
__host__ __device__ inline int varPsfAxis(int i, float v, float centre, float gap, int dim)
{
	const float t = static_cast<float>(fabs((i + 0.5) * static_cast<double>(v) - centre));
	const int a = static_cast<int>(roundf(fabsf(t) / gap));
	return a >= dim ? dim - 1 : a;
}

constexpr int kVarMaxSeg = 48;   // segments of the x axis in the launch parameters
constexpr int kVarMaxHx = 8;     // largest half size along x of the register window
constexpr int kVarOut = 8;       // outputs per thread
constexpr int kVarTileX = 32, kVarTileY = 32, kVarThreads = 256;
constexpr size_t kVarMaxShared = 113 * 1024;  // two blocks per SM

// Segments of constant LUT coordinate along one axis, of the circular axis
// unrolled to [-H, n + H): segment s covers [start[s], start[s + 1]) and holds
// its kernels' LUT offset (the coordinate times the axis' LUT stride).
struct VarSegs
{
	int n;
	short start[kVarMaxSeg + 1];
	int lut[kVarMaxSeg];
};

struct VarTile
{
	const float4* w;   // all kernels' weights, rows padded to 4 floats
	const int4* meta;  // per kernel: offset into w (float4), half sizes x, y, z
	int Hx, Hy, Hz;    // largest half sizes
	int zt;            // planes per tile
	int zTiles;        // tiles per frame
	int chunks;        // chunks of x
	VarSegs x, y, z;
	short chunkBase[kVarMaxSeg + 1];  // forward: chunks of x before each segment
};

// Adds one kernel's rows dz0 .. dz1, dy0 .. dy1 (inclusive) to the thread's
// outputs.  centre points at x0 in the thread's own row, w at the kernel's
// first row of taps; the weights of the next row are read while this one is
// added.  MASK: the window elements whose bit is clear count as 0 (elements
// of another segment; the weights are finite, checked when the LUT is made).
template <int HX, bool ADJ, bool MASK>
__device__ __forceinline__ void varBox(const float* centre, int pitch, int planePitch,
                                       const float4* __restrict__ w, int hy, int hz, int dz0,
                                       int dz1, int dy0, int dy1, unsigned mask,
                                       float (&acc)[kVarOut])
{
	constexpr int NT = 2 * HX + 1, NW = (NT + 3) / 4, NI = kVarOut + 2 * HX;
	if (dz0 > dz1 || dy0 > dy1)
		return;
	const int rows = 2 * hy + 1;
	float4 nxt[NW];
	const float4* wr = w + ((dz0 + hz) * rows + dy0 + hy) * NW;
#pragma unroll
	for (int i = 0; i < NW; i++)
		nxt[i] = __ldg(wr + i);
	for (int dz = dz0; dz <= dz1; dz++)
		for (int dy = dy0; dy <= dy1; dy++)
		{
			float in[NI], wt[4 * NW];
#pragma unroll
			for (int i = 0; i < NW; i++)
			{
				wt[4 * i] = nxt[i].x;
				wt[4 * i + 1] = nxt[i].y;
				wt[4 * i + 2] = nxt[i].z;
				wt[4 * i + 3] = nxt[i].w;
			}
			// The row after this one (past the last one: this one again).
			const int ndy = dy < dy1 ? dy + 1 : dy0;
			const int ndz = dy < dy1 ? dz : min(dz + 1, dz1);
			wr = w + ((ndz + hz) * rows + ndy + hy) * NW;
#pragma unroll
			for (int i = 0; i < NW; i++)
				nxt[i] = __ldg(wr + i);
			const int at = dz * planePitch + dy * pitch;
			const float* row = centre + (ADJ ? -at : at) - HX;
#pragma unroll
			for (int i = 0; i < NI; i++)
				in[i] = (!MASK || (mask & (1u << i))) ? row[i] : 0.f;
#pragma unroll
			for (int kk = 0; kk < NT; kk++)
#pragma unroll
				for (int m = 0; m < kVarOut; m++)
					acc[m] = __fadd_rn(
					    acc[m], __fmul_rn(in[ADJ ? m + 2 * HX - kk : m + kk], wt[kk]));
		}
}

// varBox for the run-time half size hx <= kVarMaxHx; lo, hi: bounds of the
// segment relative to x0 (MASK).
template <bool ADJ, bool MASK>
__device__ __forceinline__ void varBoxAny(const float* centre, int pitch, int planePitch,
                                          const float4* w, const int4& m, int dz0, int dz1,
                                          int dy0, int dy1, int lo, int hi, float (&acc)[kVarOut])
{
	unsigned mask = 0u;
	if constexpr (MASK)
	{
		// Bits [lo + hx, hi + hx) of the window's elements x0 - hx ...
		const int a = max(lo + m.y, 0), b = min(hi + m.y, 31);
		mask = b > a ? ((1u << b) - 1u) & ~((1u << a) - 1u) : 0u;
		if (mask == 0u)
			return;
	}
	switch (m.y)
	{
#define YRTB_VAR_CASE(N)                                                                     \
	case N:                                                                                  \
		varBox<N, ADJ, MASK>(centre, pitch, planePitch, w, m.z, m.w, dz0, dz1, dy0, dy1,     \
		                     mask, acc);                                                     \
		break;
		YRTB_VAR_CASE(0)
		YRTB_VAR_CASE(1)
		YRTB_VAR_CASE(2)
		YRTB_VAR_CASE(3)
		YRTB_VAR_CASE(4)
		YRTB_VAR_CASE(5)
		YRTB_VAR_CASE(6)
		YRTB_VAR_CASE(7)
		YRTB_VAR_CASE(8)
#undef YRTB_VAR_CASE
	default: break;
	}
}

// First and last segments that [a, b] touches.
__device__ __forceinline__ void varSpan(const VarSegs& S, int a, int b, int& s0, int& s1)
{
	s0 = 0;
	while (s0 + 1 < S.n && S.start[s0 + 1] <= a)
		s0++;
	s1 = s0;
	while (s1 + 1 < S.n && S.start[s1 + 1] <= b)
		s1++;
}

__host__ __device__ inline int varPitch(int Hx)
{
	return (kVarTileX + 2 * Hx) | 1;  // odd: the 32 rows of a warp fall in 32 banks
}

// Shared memory of a block: the tile and one staging row of outputs per thread.
__host__ __device__ inline size_t varShared(const VarTile& T)
{
	const size_t pz = T.zt + 2 * T.Hz, py = kVarTileY + 2 * T.Hy;
	return (pz * py * varPitch(T.Hx) + kVarThreads * (kVarOut + 1)) * sizeof(float);
}

__device__ __forceinline__ int varWrap(int i, int n)
{
	i %= n;
	return i < 0 ? i + n : i;
}

template <bool ADJ>
__global__ void __launch_bounds__(kVarThreads, 2)
    k_varpsf_tile(const float* __restrict__ src, float* __restrict__ dst, int nx, int ny, int nz,
                  const __grid_constant__ VarTile T)
{
	extern __shared__ float varTile[];
	const int pitch = varPitch(T.Hx);
	const int py = kVarTileY + 2 * T.Hy, pz = T.zt + 2 * T.Hz;
	float* tile = varTile;
	float* stage = tile + pz * py * pitch;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	constexpr int kWarps = kVarThreads / 32, kChunks = kVarTileX / kVarOut;

	// First output x and length of chunk c, and its segment.
	auto chunkOf = [&](int c, int& x0, int& len, int& seg)
	{
		if constexpr (ADJ)
		{
			x0 = c * kVarOut;
			len = min(kVarOut, nx - x0);
			seg = 0;
		}
		else
		{
			seg = 0;
			while (seg + 1 < T.x.n && c >= T.chunkBase[seg + 1])
				seg++;
			x0 = T.x.start[seg] + (c - T.chunkBase[seg]) * kVarOut;
			len = min(kVarOut, T.x.start[seg + 1] - x0);
		}
	};
	int tx0, len0, seg0;
	chunkOf(blockIdx.x * kChunks, tx0, len0, seg0);
	const int ty0 = blockIdx.y * kVarTileY;
	const int frame = blockIdx.z / T.zTiles;
	const int tz0 = (blockIdx.z - frame * T.zTiles) * T.zt;
	const int64_t plane = static_cast<int64_t>(nx) * ny;
	const float* in = src + frame * plane * nz;

	// Fill the tile (circular borders) and the LUT offsets of its rows.
	const int px = kVarTileX + 2 * T.Hx;
	for (int r = warp; r < pz * py; r += kWarps)
	{
		const int rz = r / py, ry = r - rz * py;
		const float* g = in + varWrap(tz0 + rz - T.Hz, nz) * plane +
		                 static_cast<int64_t>(varWrap(ty0 + ry - T.Hy, ny)) * nx;
		for (int x = lane; x < px; x += 32)
			tile[r * pitch + x] = __ldg(g + varWrap(tx0 + x - T.Hx, nx));
	}
	__syncthreads();

	float* mine = stage + warp * 32 * (kVarOut + 1);
	for (int task = warp; task < kChunks * T.zt; task += kWarps)
	{
		const int c = blockIdx.x * kChunks + task % kChunks;
		const int zl = task / kChunks;
		if (c >= T.chunks || tz0 + zl >= nz)
			continue;  // uniform over the warp
		int x0, len, seg;
		chunkOf(c, x0, len, seg);
		float acc[kVarOut];
#pragma unroll
		for (int m = 0; m < kVarOut; m++)
			acc[m] = 0.f;
		const float* centre = tile + ((zl + T.Hz) * py + lane + T.Hy) * pitch + (x0 - tx0) + T.Hx;
		const int y = ty0 + lane, z = tz0 + zl;
		if (y < ny)
		{
			int y0, y1, z0, z1;
			if constexpr (!ADJ)
			{
				varSpan(T.y, y, y, y0, y1);
				varSpan(T.z, z, z, z0, z1);
				const int4 m = __ldg(T.meta + T.x.lut[seg] + T.y.lut[y0] + T.z.lut[z0]);
				varBoxAny<false, false>(centre, pitch, py * pitch, T.w + m.x, m, -m.w, m.w, -m.z,
				                        m.z, 0, 0, acc);
			}
			else
			{
				// The kernels of the segments that the window touches, each on
				// the rows (and, where the window leaves the segment, the
				// elements) of its own sources: source p - d in the segment.
				int x1, xs;
				varSpan(T.x, x0 - T.Hx, x0 + kVarOut - 1 + T.Hx, xs, x1);
				varSpan(T.y, y - T.Hy, y + T.Hy, y0, y1);
				varSpan(T.z, z - T.Hz, z + T.Hz, z0, z1);
				for (int zs = z0; zs <= z1; zs++)
					for (int ys = y0; ys <= y1; ys++)
						for (int s = xs; s <= x1; s++)
						{
							const int4 m =
							    __ldg(T.meta + T.x.lut[s] + T.y.lut[ys] + T.z.lut[zs]);
							const int dz0 = max(-m.w, z - T.z.start[zs + 1] + 1);
							const int dz1 = min(m.w, z - T.z.start[zs]);
							const int dy0 = max(-m.z, y - T.y.start[ys + 1] + 1);
							const int dy1 = min(m.z, y - T.y.start[ys]);
							if (xs == x1)
								varBoxAny<true, false>(centre, pitch, py * pitch, T.w + m.x, m,
								                       dz0, dz1, dy0, dy1, 0, 0, acc);
							else
								varBoxAny<true, true>(centre, pitch, py * pitch, T.w + m.x, m,
								                      dz0, dz1, dy0, dy1, T.x.start[s] - x0,
								                      T.x.start[s + 1] - x0, acc);
						}
			}
		}
		// Rows of 8 outputs through shared memory: each store instruction
		// writes 4 rows of 8 consecutive x.
#pragma unroll
		for (int m = 0; m < kVarOut; m++)
			mine[lane * (kVarOut + 1) + m] = acc[m];
		__syncwarp();
		float* out = dst + (static_cast<int64_t>(frame) * nz + tz0 + zl) * plane;
#pragma unroll
		for (int k = 0; k < kVarOut; k++)
		{
			const int r = k * (32 / kVarOut) + lane / kVarOut, x = lane % kVarOut;
			if (ty0 + r < ny && x < len)
				out[static_cast<int64_t>(ty0 + r) * nx + x0 + x] = mine[r * (kVarOut + 1) + x];
		}
		__syncwarp();
	}
}

}  // namespace yrtb
