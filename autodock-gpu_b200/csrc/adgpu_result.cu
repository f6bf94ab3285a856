// adgpu_result.cu -- result processing on the device (include/adgpu_b200.h,
// "Result processing"): each run's final population ordered by energy, poses
// rebuilt from genotypes and re-scored with the reference's host scorer, the
// RMSD from the input ligand, and the runs clustered by RMSD.
//
// This file is compiled without flush-to-zero and without multiply-add
// contraction (build.py): its single- and double-precision arithmetic is the
// IEEE arithmetic of the reference's host code, which it follows operation by
// operation, in the same order, so that the energies, RMSDs and cluster
// assignments are the ones the reference's process_result computes.  The one
// source of difference is the double-precision sin/cos of the pose builder,
// which may round differently from the host's libm in the last place.
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>
#include "adgpu_prep.h"
#include "adgpu_result.h"
#include "adgpu_tables.h"
#include "adgpu_nvtx.h"

namespace adgpu {
namespace {

constexpr int kTab = 2048;                 // IntraTables distance tables, 0.01..20.48 A
constexpr int kWarps = 4;                  // rescoring warps per CTA
constexpr double kPi = 3.14159265359;      // PI, host/inc/miscellaneous.h:51
constexpr float kGbond = 50.0f;            // G, common/defines.h:108
constexpr int kCG = 24, kG0 = 25;          // ATYPE_CG_IDX, ATYPE_G0_IDX, common/defines.h:71-72
constexpr float kOutOfGridTol = 0.0005f;   // outofgrid_tolerance of make_resfiles' calc_interE_f calls
constexpr float kDcutoff = 8.0f;           // dcutoff of make_resfiles' calc_intraE_f calls

struct PostDev {
	int N, NL, NR, NT, Q, P;
	int gx, gy, gz, nmaps;                 // grid points, type maps
	int rmsd_atoms, symmetry, rescore_all;
	int cells;                             // grid layout: 0 reference (4 floats per point per map), 1 cell records
	const float* grid;
	int flex_or_cg;                        // some pair adds to interflexE: ligand-flexres or CG-G0
	const double *ref_xyz, *input_xyz, *charge, *rot_move, *rot_unit;
	const unsigned long long* rot_mask;
	const float4* rtab;                    // (1/r^6, 1/r^10, 1/r^12, -) of the distance tables
	const float2* etab;                    // (elec factor, desolvation gaussian)
	const int *type, *map;
	const unsigned char* ignore;
	const struct PostPair* pairs;
	double movvec[3];                      // get_movvec_to_origo of the reference orientation
	double spacing, origin[3];
	float smooth, elec_min_distance;
};

// One intramolecular contributor with its type-pair parameters and charge
// products resolved on the host in the reference's operations.
struct __align__(16) PostPair {
	double v12, vn;                        // vw_A, vw_B, or vw_C, vw_D of an H-bond pair
	float opt, q1q2, sv;                   // reqm; charge product; s1*w2 + s2*w1 of the desolvation
	unsigned int ij;                       // i | j << 8 | H-bond << 16 | CG-G0 << 17 | ligand-flexres << 18
};

struct RunRec {                            // per run, written by the rescoring of its best entity
	float inter, intraflex, intra, interflex, elec, rmsd, energy;
	float crmsd;
	int clus, subrank, output, rank;
};

// ---------------------------------------------------------------------------
// arrange_result (host/src/processresult.cpp:31-59): a stable ascending bubble
// sort of each run's entities by energy.  A NaN energy compares false both
// ways, so it never moves and the entities on either side of it are sorted
// separately; each entity's destination is its rank inside its NaN-free
// segment (ties keep their order).
// ---------------------------------------------------------------------------
template <class T>
__device__ int stable_rank(const T* e, int n, int i)
{
	const T x = e[i];
	if (isnan(x)) return i;
	int s = i;
	while (s > 0 && !isnan(e[s - 1])) s--;
	int rank = s;
	for (int j = s; j < n && !isnan(e[j]); j++) rank += (e[j] < x) || (e[j] == x && j < i);
	return rank;
}

// The rank in an array without NaN: one segment, no test per step.
template <class T>
__device__ int plain_rank(const T* e, int n, int i)
{
	const T x = e[i];
	int rank = 0;
#pragma unroll 4
	for (int j = 0; j < n; j++) rank += (e[j] < x) || (e[j] == x && j < i);
	return rank;
}

// V: float4, or float for populations that are not 16-byte aligned.
template <class V>
__global__ void __launch_bounds__(256) arrange_kernel(float* pop, float* energies, float* scratch, int P)
{
	constexpr int kPer = 64 * (int)sizeof(float) / (int)sizeof(V);      // of a genotype
	extern __shared__ float sh_e[];
	int* dst = reinterpret_cast<int*>(sh_e + P);
	const size_t r = blockIdx.x;
	float* E = energies + r * P;
	V* G = reinterpret_cast<V*>(pop + r * P * 64);
	V* S = reinterpret_cast<V*>(scratch + r * P * 64);
	int nans = 0;
	for (int i = threadIdx.x; i < P; i += blockDim.x) {
		const float e = E[i];
		sh_e[i] = e;
		nans |= isnan(e);
	}
	nans = __syncthreads_or(nans);
	for (int i = threadIdx.x; i < P; i += blockDim.x) dst[i] = nans ? stable_rank(sh_e, P, i) : plain_rank(sh_e, P, i);
	__syncthreads();
	for (int k = threadIdx.x; k < P * kPer; k += blockDim.x) S[dst[k / kPer] * kPer + k % kPer] = G[k];
	for (int i = threadIdx.x; i < P; i += blockDim.x) E[dst[i]] = sh_e[i];
	__syncthreads();
	for (int k = threadIdx.x; k < P * kPer; k += blockDim.x) G[k] = S[k];
}

// ---------------------------------------------------------------------------
// Pose building: change_conform (host/src/processligand.cpp:1607-1664) with
// rotate (host/src/miscellaneous.cpp:150-256): the point is moved by
// -movvec, turned by the quaternion q = (cos a/2, sin a/2 n) as q v q^-1
// (the products written out with v's and the result's scalar parts zero),
// and moved back.
// ---------------------------------------------------------------------------
__device__ void rotate_point(double p[3], const double mv[3], const double n[3], double c, double s)
{
	p[0] = p[0] - mv[0];
	p[1] = p[1] - mv[1];
	p[2] = p[2] - mv[2];
	const double lq = c, lx = s * n[0], ly = s * n[1], lz = s * n[2];
	const double rq = lq, rx = -1 * lx, ry = -1 * ly, rz = -1 * lz;
	const double tq = 0 - lx * p[0] - ly * p[1] - lz * p[2];
	const double tx = lq * p[0] + 0 + ly * p[2] - lz * p[1];
	const double ty = lq * p[1] - lx * p[2] + 0 + lz * p[0];
	const double tz = lq * p[2] + lx * p[1] - ly * p[0] + 0;
	p[0] = tq * rx + tx * rq + ty * rz - tz * ry;
	p[1] = tq * ry - tx * rz + ty * rq + tz * rx;
	p[2] = tq * rz + tx * ry - ty * rx + tz * rq;
	p[0] = p[0] + mv[0];
	p[1] = p[1] + mv[1];
	p[2] = p[2] + mv[2];
}

__device__ __forceinline__ double dist2(const double* a, const double* b)
{
	const double s1 = a[0] - b[0], s2 = a[1] - b[1], s3 = a[2] - b[2];
	return s1 * s1 + s2 * s2 + s3 * s3;
}

// calc_rmsd (host/src/processligand.cpp:1441-1489) of pose xyz against ref:
// with symmetry, each atom's squared distance to the nearest reference atom
// of its type (100000 when there is none).  Per-atom terms in parallel into
// the warp's scratch `terms` (n doubles), the sum in atom order on lane 0,
// the result broadcast to the warp.
__device__ double warp_rmsd(const double* xyz, const double* ref, const int* type, int n, int symmetry, int lane,
                            double* terms)
{
	for (int a = lane; a < n; a += 32) {
		double m;
		if (symmetry) {
			const int ta = type[a];
			m = 100000;
			for (int b = 0; b < n; b++)
				if (ta == type[b]) {
					const double d2 = dist2(xyz + 3 * a, ref + 3 * b);
					if (d2 < m) m = d2;
				}
		} else m = dist2(xyz + 3 * a, ref + 3 * a);
		terms[a] = m;
	}
	__syncwarp();
	double sum = 0.0;
	if (lane == 0)
		for (int a = 0; a < n; a++) sum += terms[a];
	__syncwarp();
	return __shfl_sync(0xffffffffu, sqrt(sum / (unsigned)n), 0);
}

// ---------------------------------------------------------------------------
// Re-scoring, one warp per entity: the per-entity body of make_resfiles
// (host/src/processresult.cpp:421-475): change_conform_f, calc_interE_f in
// grid units, scale_ligand to Angstrom, calc_intraE_f, move_ligand to the
// grid's origin, calc_rmsd.  Per-atom and per-pair terms are computed by the
// lanes, and each energy is summed by one lane in the reference's atom and
// pair order, so the float sums round as the host's do.  A term that the
// reference does not add to a sum is staged as +0, which leaves the sum as it
// is.  What bounds it: those sums are the only serial part, so the lanes stage
// 32 entries of each sum in shared memory (rows of 36 floats: four rows read
// by four lanes fall in different banks) and one lane per sum reads them four
// at a time, about 45 instructions for 32 pairs.  (Handing every term to lane
// 0 by shuffles took five shuffles and the branches of the accumulators for
// each pair, 600 instructions for 32 pairs.)  15,000 entities of the 45-atom,
// 777-pair ligand: 0.75 ms before; the whole call 5.48 -> 0.71 ms on B200, of
// which the clustering was 4.2 ms.
// ---------------------------------------------------------------------------
constexpr int kRow = 36;                   // floats of a staged row
constexpr int kRows = 5;

// Adds row `lane`'s 32 staged terms, in order, to the lane's sum (lanes 0..nsum-1).
__device__ __forceinline__ void add_row(const float* st, int lane, int nsum, float& sum)
{
	if (lane >= nsum) return;
	const float4* row = reinterpret_cast<const float4*>(st + lane * kRow);
	for (int k = 0; k < 8; k++) {
		const float4 v = row[k];
		sum += v.x; sum += v.y; sum += v.z; sum += v.w;
	}
}

__host__ __device__ constexpr size_t rescore_warp_bytes(int N, int NR)
{
	// coordinates, sines and cosines, per-atom RMSD terms; staged rows
	return ((size_t)(4 * N + 2 * NR + 8) * sizeof(double) + 15) / 16 * 16 + (size_t)kRows * kRow * sizeof(float);
}

__global__ void __launch_bounds__(kWarps * 32)
rescore_kernel(PostDev D, const float* pop, const float* energies, int ntask, RunRec* runs, double* best_xyz,
               float* peratom, float* entities)
{
	extern __shared__ __align__(16) unsigned char sh_w[];
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int N = D.N, NL = D.NL, NR = D.NR;
	const size_t wb = rescore_warp_bytes(N, NR);
	double* xyz = reinterpret_cast<double*>(sh_w + (size_t)warp * wb);
	double* trig = xyz + 3 * N;                // cos, sin of each torsion's half angle; genrot axis, cos, sin
	double* terms = trig + 2 * NR + 8;         // N
	float* st = reinterpret_cast<float*>(sh_w + (size_t)(warp + 1) * wb) - kRows * kRow;
	const size_t g3_4 = ((size_t)D.gx * D.gy * D.gz) << 2;
	for (int task = blockIdx.x * kWarps + warp; task < ntask; task += gridDim.x * kWarps) {
		const int run = D.rescore_all ? task / D.P : task;
		const int ent = D.rescore_all ? task % D.P : 0;
		const float* g = pop + ((size_t)run * D.P + ent) * 64;
		// half-angle sines and cosines (rotate computes them per call; same values)
		for (int rb = lane; rb < NR; rb += 32) {
			const double ang = (double)g[6 + rb];
			const double half = ang / 2 / 180 * kPi;
			trig[2 * rb] = cos(half);
			trig[2 * rb + 1] = sin(half);
		}
		if (lane == 0) {
			const double phi = ((double)g[3]) / 180 * kPi, theta = ((double)g[4]) / 180 * kPi;
			double* gr = trig + 2 * NR;
			gr[0] = sin(theta) * cos(phi);
			gr[1] = sin(theta) * sin(phi);
			gr[2] = cos(theta);
			const double half = (double)g[5] / 2 / 180 * kPi;
			gr[3] = cos(half);
			gr[4] = sin(half);
		}
		__syncwarp();
		const double* gr = trig + 2 * NR;
		const double zero[3] = {0.0, 0.0, 0.0};
		for (int a = lane; a < N; a += 32) {
			double p[3] = {D.ref_xyz[3 * a], D.ref_xyz[3 * a + 1], D.ref_xyz[3 * a + 2]};
			if (a < NL) for (int k = 0; k < 3; k++) p[k] += D.movvec[k];
			const unsigned long long m = D.rot_mask[a];
			for (int rb = 0; rb < NR; rb++)
				if ((m >> rb) & 1ull) rotate_point(p, D.rot_move + 3 * rb, D.rot_unit + 3 * rb, trig[2 * rb], trig[2 * rb + 1]);
			if (a < NL) {
				rotate_point(p, zero, gr, gr[3], gr[4]);
				for (int k = 0; k < 3; k++) p[k] += (double)g[k];
			}
			for (int k = 0; k < 3; k++) xyz[3 * a + k] = p[k];
		}
		__syncwarp();

		// calc_interE_f (host/src/processligand.cpp:1796-2055)
		const bool best = ent == 0;
		float isum = 0.0f;                     // lane 0: interE, lane 1: intraflexE, lane 2: elecE
		for (int base = 0; base < N; base += 32) {
			const int a = base + lane;
			int kind = 0;                      // 0: not counted, 1: outside the grid, 2: interpolated
			float val = 0.0f, vd = 0.0f, e = 0.0f;   // vd: vdW + desolvation (the per-atom vdW the reference reports)
			if (a < N && !D.ignore[a]) {
				float x = (float)xyz[3 * a], y = (float)xyz[3 * a + 1], z = (float)xyz[3 * a + 2];
				const float q = (float)D.charge[a];
				const float X1 = (float)(D.gx - 1), Y1 = (float)(D.gy - 1), Z1 = (float)(D.gz - 1);
				bool out = x < 0 || x >= X1 || y < 0 || y >= Y1 || z < 0 || z >= Z1;
				if (out) {
					if (x < 0) x += kOutOfGridTol;
					if (y < 0) y += kOutOfGridTol;
					if (z < 0) z += kOutOfGridTol;
					if (x >= X1) x -= kOutOfGridTol;
					if (y >= Y1) y -= kOutOfGridTol;
					if (z >= Z1) z -= kOutOfGridTol;
					out = x < 0 || x >= X1 || y < 0 || y >= Y1 || z < 0 || z >= Z1;
				}
				if (out) {
					val += 16777216;
					kind = 1;
				} else {
					const int xl = (int)floorf(x), yl = (int)floorf(y), zl = (int)floorf(z);
					// the 8 corner values of each map in idx_000 .. idx_111 order: 8 consecutive
					// floats from the point in the reference layout; the cell's record (e, d,
					// type maps) in the engine's layout, the same values in the same order
					const float *cv, *ce, *cd;
					if (D.cells) {
						const float* rec = D.grid + (size_t)(xl + yl * (D.gx - 1) + zl * (D.gx - 1) * (D.gy - 1)) *
						                            (size_t)(D.nmaps + 2) * 8;
						cv = rec + (size_t)(2 + D.map[a]) * 8;
						ce = rec;
						cd = rec + 8;
					} else {
						const float* c0 = D.grid + ((size_t)(unsigned)(xl + yl * D.gx + zl * D.gx * D.gy) << 2);
						cv = c0 + (size_t)D.map[a] * g3_4;
						ce = c0 + (size_t)D.nmaps * g3_4;
						cd = ce + g3_4;
					}
					const float dx = x - xl, omdx = 1.0f - dx;
					const float dy = y - yl, omdy = 1.0f - dy;
					const float dz = z - zl, omdz = 1.0f - dz;
					float w[8];
					w[0] = omdx * omdy * omdz; w[1] = omdx * dy * omdz; w[2] = omdx * omdy * dz; w[3] = omdx * dy * dz;
					w[4] = dx * omdy * omdz;   w[5] = dx * dy * omdz;   w[6] = dx * omdy * dz;   w[7] = dx * dy * dz;
					auto interp = [&](const float* c) {
						return c[0] * w[0] + c[1] * w[1] + c[2] * w[2] + c[3] * w[3] + c[4] * w[4] + c[5] * w[5] +
						       c[6] * w[6] + c[7] * w[7];
					};
					const float v = interp(cv);
					val += v;
					e = q * interp(ce);
					val += e;
					const float ed = fabsf(q) * interp(cd);
					val += ed;
					// AD4_desolv_peratom_vdW is defined (host/src/processligand.cpp:30, 2041-2043)
					vd = v + ed;
					kind = 2;
				}
			}
			if (best && a < N) {
				float* pa = peratom + ((size_t)run * N + a) * 2;
				pa[0] = kind == 2 ? vd : (kind == 1 ? 100000.0f : 0.0f);
				pa[1] = kind == 2 ? e : (kind == 1 ? 100000.0f : 0.0f);
			}
			const bool lig = a < NL;
			st[lane] = kind && lig ? val : 0.0f;
			st[kRow + lane] = kind && !lig ? val : 0.0f;
			st[2 * kRow + lane] = kind == 2 && lig ? e : 0.0f;
			__syncwarp();
			add_row(st, lane, 3, isum);
			__syncwarp();
		}
		const float interE = __shfl_sync(0xffffffffu, isum, 0);
		const float intraflexE = __shfl_sync(0xffffffffu, isum, 1);
		const float elecE = __shfl_sync(0xffffffffu, isum, 2);

		// scale_ligand to Angstrom (the grid's spacing)
		for (int a = lane; a < N; a += 32)
			for (int k = 0; k < 3; k++) xyz[3 * a + k] *= D.spacing;
		__syncwarp();

		// calc_intraE_f (host/src/processligand.cpp:2058-2331), without
		// modified pairs (the front end has none) and without contact analysis
		float psum = 0.0f;                     // lane 0: vW, lane 1: elec, lane 2: desolv, lane 3: interflexE
		const float delta = 0.5f * D.smooth;
		for (int base = 0; base < D.Q; base += 32) {
			const int pi = base + lane;
			bool flex = false;
			float t_cg = 0.0f, t_vdw = 0.0f, t_a = 0.0f, t_b = 0.0f;
			if (pi < D.Q) {
				const PostPair pp = D.pairs[pi];
				const int i = (int)(pp.ij & 0xFFu), j = (int)((pp.ij >> 8) & 0xFFu);
				flex = (pp.ij >> 18) & 1u;
				float dist = (float)sqrt(dist2(xyz + 3 * i, xyz + 3 * j));
				int did = (int)floorf((100.0f * dist) + 0.5f) - 1;
				if (did < 0) did = 0;
				if ((pp.ij >> 17) & 1u) t_cg = kGbond * dist;
				if (dist < kDcutoff) {
					const float opt = pp.opt;
					float sd;
					if (dist <= (opt - delta)) sd = dist + delta;
					else if (dist < (opt + delta)) sd = opt;
					else sd = dist - delta;
					int sid = (int)floorf((100.0f * sd) + 0.5f) - 1;
					if (sid < 0) sid = 0;
					const float4 rt = D.rtab[sid];
					const float vdw1 = (float)(pp.v12 * rt.z);
					const float vdw2 = (float)(pp.vn * ((pp.ij >> 16) & 1u ? rt.y : rt.x));
					t_vdw = vdw1 - vdw2;
				}
				if (dist < 20.48) {
					int eid = did;
					if (dist < D.elec_min_distance) {
						dist = D.elec_min_distance;
						eid = (int)floor((100 * dist) + 0.5) - 1;
						// the reference reads outside its table here when elec_min_distance < 0.005
						eid = eid < 0 ? 0 : (eid >= kTab ? kTab - 1 : eid);
					}
					const float2 et = D.etab[eid];
					t_a = pp.q1q2 * et.x;
					t_b = pp.sv * et.y;
				}
			}
			// a ligand-flexres pair's terms go to interflexE, all but its CG-G0
			// term, which goes the other way round (host/src/processligand.cpp:2142-2145)
			st[lane] = flex ? t_cg : t_vdw;
			st[kRow + lane] = flex ? 0.0f : t_a;
			st[2 * kRow + lane] = flex ? 0.0f : t_b;
			if (D.flex_or_cg) {
				st[3 * kRow + lane] = flex ? t_vdw : t_cg;
				st[4 * kRow + lane] = flex ? t_a + t_b : 0.0f;
			}
			__syncwarp();
			add_row(st, lane, 3, psum);
			if (D.flex_or_cg && lane == 3)
				for (int k = 0; k < 32; k++) { psum += st[3 * kRow + k]; psum += st[4 * kRow + k]; }
			__syncwarp();
		}
		const float vW = __shfl_sync(0xffffffffu, psum, 0), el = __shfl_sync(0xffffffffu, psum, 1);
		const float desolv = __shfl_sync(0xffffffffu, psum, 2), interflexE = __shfl_sync(0xffffffffu, psum, 3);
		const float intraE = vW + el + desolv;

		// move_ligand by the grid's origin (ligand and flexible residues)
		for (int a = lane; a < N; a += 32)
			for (int k = 0; k < 3; k++) xyz[3 * a + k] += D.origin[k];
		__syncwarp();
		double rmsd = 0.0;
		if (best || D.rescore_all)
			rmsd = warp_rmsd(xyz, D.input_xyz, D.type, D.rmsd_atoms, D.symmetry, lane, terms);
		if (lane == 0) {
			if (entities) {
				float* o = entities + ((size_t)run * D.P + ent) * 3;
				o[0] = intraE + intraflexE;
				o[1] = interE + interflexE;
				o[2] = (float)rmsd;
			}
			if (best) {
				RunRec& R = runs[run];
				R.inter = interE; R.intraflex = intraflexE; R.intra = intraE; R.interflex = interflexE;
				R.elec = elecE; R.rmsd = (float)rmsd; R.energy = energies[(size_t)run * D.P];
				R.crmsd = 0.0f; R.clus = 0; R.subrank = 0; R.output = 1; R.rank = 0;
			}
		}
		if (best)
			for (int a = lane; a < N; a += 32)
				for (int k = 0; k < 3; k++) best_xyz[((size_t)run * N + a) * 3 + k] = xyz[3 * a + k];
		__syncwarp();
	}
}

// ---------------------------------------------------------------------------
// generate_output's ordering and clustering (host/src/processresult.cpp:
// 688-804): runs ordered by energy (inter + interflex, plus intra terms for
// flexible residues alone) with the same NaN-segment stable ranking; then
// each run in that order joins the first cluster whose centre (its first
// member) lies within the RMSD tolerance, or founds a new one.
//
// The scan over runs is serial, so what it needs per run is made small: the
// RMSDs of all pairs (later run, earlier run) are taken beforehand over the
// whole GPU (pair_rmsd_kernel), as one bit each for "within the tolerance",
// and one warp scans the rows.  Centres are founded in run order, so the first
// cluster within the tolerance is the lowest set bit of row & centres.  That
// needs R^2/2 RMSDs instead of one per run and centre, so it serves up to
// kPairRuns runs (4 MB of RMSDs); above it cluster_kernel takes the RMSDs to
// the current centres as it goes, one warp per centre.
// ---------------------------------------------------------------------------
constexpr int kPairRuns = 1024;

__device__ double run_energy(const RunRec& r, int free_roaming)
{
	double e = (double)(r.inter + r.interflex);
	if (!free_roaming) e += (double)(r.intra + r.intraflex);
	return e;
}

// Energy order of the runs.  Launch with 1024 threads.
__global__ void __launch_bounds__(1024) order_kernel(int R, RunRec* runs, double* en, int* order, int free_roaming)
{
	__shared__ double s_en[kPairRuns];
	const int tid = threadIdx.x;
	double* const E = R <= kPairRuns ? s_en : en;
	int nans = 0;
	for (int r = tid; r < R; r += blockDim.x) {
		E[r] = run_energy(runs[r], free_roaming);
		nans |= isnan(E[r]);
	}
	nans = __syncthreads_or(nans);
	for (int r = tid; r < R; r += blockDim.x) {
		const int rank = nans ? stable_rank(E, R, r) : plain_rank(E, R, r);
		order[rank] = r;
		runs[r].rank = rank;
	}
}

// RMSD of the w-th run in energy order from the u-th, u < w, for every pair
// p = w (w - 1) / 2 + u: one warp each.
__global__ void __launch_bounds__(kWarps * 32)
pair_rmsd_kernel(PostDev D, int R, const double* best_xyz, const int* order, double tol, float* mat, unsigned int* bits)
{
	extern __shared__ __align__(16) unsigned char sh_w[];
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n = D.rmsd_atoms, N = D.N, W = (R + 31) / 32;
	double* terms = reinterpret_cast<double*>(sh_w) + (size_t)warp * N;
	const int npair = R * (R - 1) / 2;
	for (int p = blockIdx.x * kWarps + warp; p < npair; p += gridDim.x * kWarps) {
		int w = (int)((1.0 + sqrt(1.0 + 8.0 * (double)p)) * 0.5);
		while (w * (w - 1) / 2 > p) w--;
		while (w * (w + 1) / 2 <= p) w++;
		const int u = p - w * (w - 1) / 2;
		const double d = warp_rmsd(best_xyz + (size_t)order[w] * N * 3, best_xyz + (size_t)order[u] * N * 3, D.type, n,
		                           D.symmetry, lane, terms);
		if (lane == 0) {
			mat[(size_t)w * R + u] = (float)d;
			if (d <= tol) atomicOr(bits + (size_t)w * W + (u >> 5), 1u << (u & 31));
		}
		__syncwarp();
	}
}

// Cluster statistics of cluster c (host/src/processresult.cpp:748-804), its
// members in energy order; clus_of(u) is the cluster of the u-th run in order.
template <class F>
__device__ void cluster_stats(int c, int R, RunRec* runs, const int* order, int ncp, int free_roaming, double torsional,
                              adgpu_cluster* clusters, F clus_of)
{
	int sub = 0;
	double sum = 0.0, bestE = 0.0;
	int best_run = 0;
	for (int u = 0; u < R; u++) {
		if (clus_of(u) != c + 1) continue;
		const int j = order[u];
		sub++;
		sum += runs[j].inter + runs[j].interflex + torsional;
		if (!free_roaming) sum += runs[j].intra + runs[j].intraflex;
		runs[j].subrank = sub;
		runs[j].output = !((ncp > 0) && (sub > ncp)) && (ncp >= 0);
		if (sub == 1) {
			bestE = runs[j].inter + runs[j].interflex + torsional;
			if (!free_roaming) bestE += runs[j].intra + runs[j].intraflex;
			best_run = j + 1;
			runs[j].output = 1;
		}
	}
	clusters[c].size = sub;
	clusters[c].best_run = best_run;
	clusters[c].best_energy = bestE;
	clusters[c].sum_energy = sum;
}

// The scan over the rows of pair_rmsd_kernel and the cluster statistics, R <=
// kPairRuns.  Dynamic shared memory: the rows.
__global__ void __launch_bounds__(256)
cluster_scan_kernel(int R, RunRec* runs, const int* order, const float* mat, const unsigned int* bits, int ncp,
                    int free_roaming, double torsional, adgpu_cluster* clusters, int* nclus)
{
	extern __shared__ unsigned int s_bits[];
	__shared__ short s_clus[kPairRuns], s_centre[kPairRuns];
	__shared__ int s_K;
	const int tid = threadIdx.x, lane = tid & 31, W = (R + 31) / 32;
	for (int k = tid; k < R * W; k += blockDim.x) s_bits[k] = bits[k];
	__syncthreads();
	if (tid < 32) {
		unsigned int centres = 0;          // lane l: runs 32 l .. 32 l + 31
		int K = 0;
		for (int w = 0; w < R; w++) {
			const unsigned int m = lane < W ? s_bits[w * W + lane] & centres : 0u;
			const unsigned int any = __ballot_sync(0xffffffffu, m != 0u);
			int u = w;
			if (any) {
				const int l = __ffs(any) - 1;
				u = 32 * l + __ffs(__shfl_sync(0xffffffffu, m, l)) - 1;
			} else {
				K++;
				if (lane == (w >> 5)) centres |= 1u << (w & 31);
			}
			if (lane == 0) {
				s_centre[w] = (short)u;
				s_clus[w] = u == w ? (short)K : s_clus[u];
			}
		}
		if (lane == 0) s_K = K;
	}
	__syncthreads();
	for (int w = tid; w < R; w += blockDim.x) {
		RunRec& r = runs[order[w]];
		r.clus = s_clus[w];
		r.crmsd = s_centre[w] == w ? 0.0f : mat[(size_t)w * R + s_centre[w]];
	}
	const int K = s_K;
	for (int c = tid; c < K; c += blockDim.x)
		cluster_stats(c, R, runs, order, ncp, free_roaming, torsional, clusters, [&](int u) { return (int)s_clus[u]; });
	if (tid == 0) *nclus = K;
}

// More than kPairRuns runs: the RMSDs to all current centres taken in
// parallel (one warp per centre) for each run in turn.  Dynamic shared memory:
// N doubles per warp.
__global__ void __launch_bounds__(1024)
cluster_kernel(PostDev D, int R, RunRec* runs, const double* best_xyz, const int* order, int* centers,
               double* crmsd, double tol, int ncp, int free_roaming, double torsional,
               adgpu_cluster* clusters, int* nclus)
{
	extern __shared__ __align__(16) unsigned char sh_w[];
	__shared__ int s_found, s_K;
	__shared__ double s_rmsd;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
	const int n = D.rmsd_atoms, N = D.N;
	double* terms = reinterpret_cast<double*>(sh_w) + (size_t)warp * N;
	if (tid == 0) {
		const int c0 = order[0];
		runs[c0].clus = 1;
		runs[c0].crmsd = 0.0f;
		centers[0] = c0;
		s_K = 1;
	}
	__syncthreads();
	for (int w = 1; w < R; w++) {
		const int i = order[w];
		const int K = s_K;
		for (int c = warp; c < K; c += nwarps) {
			const double d = warp_rmsd(best_xyz + (size_t)i * N * 3, best_xyz + (size_t)centers[c] * N * 3, D.type, n,
			                           D.symmetry, lane, terms);
			if (lane == 0) crmsd[c] = d;
			__syncwarp();
		}
		__syncthreads();
		if (tid == 0) {
			int f = -1;
			for (int c = 0; c < K; c++)
				if (crmsd[c] <= tol) { f = c; break; }
			s_found = f;
			s_rmsd = f >= 0 ? crmsd[f] : 0.0;
		}
		__syncthreads();
		if (tid == 0) {
			if (s_found >= 0) {
				runs[i].clus = s_found + 1;
				runs[i].crmsd = (float)s_rmsd;
			} else {
				centers[K] = i;
				runs[i].clus = K + 1;
				runs[i].crmsd = 0.0f;
				s_K = K + 1;
			}
		}
		__syncthreads();
	}
	const int K = s_K;
	for (int c = tid; c < K; c += blockDim.x)
		cluster_stats(c, R, runs, order, ncp, free_roaming, torsional, clusters, [&](int u) { return runs[order[u]].clus; });
	if (tid == 0) *nclus = K;
}

// IntraTables' distance tables (calc_distdep_tables_f,
// host/src/processligand.cpp:1543-1570) on the host, with the host's libm as
// the reference computes them: 1/r^6, 1/r^10, 1/r^12, the distance-dependent
// dielectric elec factor and the desolvation gaussian at r = 0.01 .. 20.48 A.
double ddd_mehler_solmajer(double d)
{
	// Mehler & Solmajer (1991) sigmoidal dielectric with AutoDock's constants
	// (host/src/processligand.cpp:1491-1512): the constants are long double
	// literals held in doubles, and the denominator is formed in long double.
	const double lambda = 0.003627L, epsilon0 = 78.4L, A = -8.5525L, rk = 7.7839L;
	const double B = epsilon0 - A;
	const double lambda_B = -lambda * B;
	const double eps = A + B / (1.0L + rk * exp(lambda_B * d));
	return eps;
}

// What the tables hold apart from the two coefficients is the same for every
// ligand and is made once.
struct DistanceTables {
	float4 r[kTab];
	double eps_r[kTab];                    // dist * dielectric
	float gauss[kTab];
	DistanceTables()
	{
		float dist = 0;
		const float sigma = 3.6f;
		for (int i = 0; i < kTab; i++) {
			dist += 0.01;
			r[i] = make_float4(1 / powf(dist, 6), 1 / powf(dist, 10), 1 / powf(dist, 12), 0.0f);
			eps_r[i] = dist * ddd_mehler_solmajer(dist);
			gauss[i] = expf(-1 * dist * dist / (2 * sigma * sigma));
		}
	}
	static const DistanceTables& get()
	{
		static const DistanceTables t;
		return t;
	}
};

template <class T>
size_t put(std::vector<unsigned char>& blob, const T* src, size_t n)
{
	size_t off = (blob.size() + 15) / 16 * 16;
	blob.resize(off + n * sizeof(T));
	if (n) memcpy(blob.data() + off, src, n * sizeof(T));
	return off;
}

// Raises a kernel's dynamic shared-memory limit.  The limit belongs to the
// function, not to a launch, so bytes is the most that any call asks for: a
// call's own size would lower the limit of one that another thread is about to
// launch.
template <class F>
cudaError_t allow_smem(F* kernel, size_t bytes)
{
	return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace
}  // namespace adgpu

using namespace adgpu;

extern "C" {

adgpu_status adgpu_result_params_default(adgpu_result_params* p)
{
	if (!p) return fail(ADGPU_ERR_ARG, "null argument");
	memset(p, 0, sizeof(*p));
	p->rmsd_tolerance = 2.0f;
	p->handle_symmetry = 1;
	p->calc_clustering = 1;
	p->nr_cluster_poses = 0;
	p->free_roaming_ligand = 1;
	p->rescore_entities = 0;
	p->coeff_tors = 0.2983;
	return ADGPU_OK;
}

}  // extern "C"

namespace adgpu {

adgpu_status process_result_core(const PostLigand& L, const uint32_t* pairs, const adgpu_dockpars& dp,
                                 const float* grid, int grid_cells, float* populations, float* energies,
                                 uint32_t num_runs, const adgpu_result_params* params, adgpu_run_result* runs_out,
                                 adgpu_cluster* clusters_out, int* num_clusters, double* best_xyz, float* peratom,
                                 float* entities, cudaStream_t st, cudaMemPool_t pool)
{
	if (!grid || !populations || !energies || !params || !runs_out || !clusters_out || !num_clusters)
		return fail(ADGPU_ERR_ARG, "null argument");
	if (num_runs == 0 || num_runs > ADGPU_MAX_RUNS) return fail(ADGPU_ERR_LIMIT, "num_runs must be 1..8192");
	if (L.natoms <= 0) return fail(ADGPU_ERR_STATE, "ligand carries no result-processing data");
	if (params->nr_cluster_poses < 0)
		return fail(ADGPU_ERR_ARG, "nr_cluster_poses < 0 (poses chosen by contact analysis) is not supported");
	if (entities && !params->rescore_entities) return fail(ADGPU_ERR_ARG, "entities output needs rescore_entities");
	const int N = L.natoms, NR = L.nrot, NT = L.ntypes, P = dp.pop_size, R = (int)num_runs;
	const int Q = dp.num_of_intraE_contributors;

	// host side: constant tables (IntraTables), the pairs and the packed ligand
	const DistanceTables& T = DistanceTables::get();
	std::vector<float2> etab(kTab);
	for (int i = 0; i < kTab; i++) etab[i] = make_float2((float)(dp.coeff_elec / T.eps_r[i]), dp.coeff_desolv * T.gauss[i]);
	std::vector<float> qabs(N);
	for (int i = 0; i < N; i++) qabs[i] = dp.qasp * fabs(L.charge[i]);        // calc_q_tables_f
	std::vector<PostPair> pp(Q);
	bool flex_or_cg = false;
	for (int k = 0; k < Q; k++) {
		const int i = (int)pairs[2 * k], j = (int)pairs[2 * k + 1], t1 = L.type[i], t2 = L.type[j], tp = t1 * NT + t2;
		const int v1 = L.vw_index[t1], v2 = L.vw_index[t2];
		const bool hb = L.is_hb[tp] != 0, cg = (v1 == kCG && v2 == kG0) || (v1 == kG0 && v2 == kCG);
		const bool flex = ((i >= L.true_lig_atoms) + (j >= L.true_lig_atoms)) & 1;
		const float s1 = (float)(L.solpar[t1] + qabs[i]), s2 = (float)(L.solpar[t2] + qabs[j]);
		const float w1 = (float)L.volume[t1], w2 = (float)L.volume[t2];
		pp[k].v12 = hb ? L.vw_C[tp] : L.vw_A[tp];
		pp[k].vn = hb ? L.vw_D[tp] : L.vw_B[tp];
		pp[k].opt = (float)L.reqm_AB[tp];
		pp[k].q1q2 = (float)((double)(float)L.charge[i] * L.charge[j]);
		pp[k].sv = s1 * w2 + s2 * w1;
		pp[k].ij = (unsigned)i | (unsigned)j << 8 | (unsigned)hb << 16 | (unsigned)cg << 17 | (unsigned)flex << 18;
		flex_or_cg |= cg || flex;
	}
	std::vector<unsigned char> blob;
	const size_t o_ref = put(blob, L.ref_xyz.data(), 3 * N), o_in = put(blob, L.input_xyz.data(), 3 * N),
	             o_q = put(blob, L.charge.data(), N), o_mv = put(blob, L.rot_move.data(), 3 * NR),
	             o_un = put(blob, L.rot_unit.data(), 3 * NR), o_mask = put(blob, L.rot_mask.data(), N),
	             o_rt = put(blob, T.r, kTab), o_et = put(blob, etab.data(), kTab), o_ty = put(blob, L.type.data(), N),
	             o_map = put(blob, L.map.data(), N), o_ig = put(blob, L.ignore_inter.data(), N),
	             o_pr = put(blob, pp.data(), Q);
	// device scratch
	const size_t n_pop = (size_t)R * P * 64;
	size_t off = (blob.size() + 255) / 256 * 256;
	auto take = [&](size_t bytes) { size_t o = off; off = (off + bytes + 255) / 256 * 256; return o; };
	const size_t o_scr = take(n_pop * 4), o_runs = take((size_t)R * sizeof(RunRec)), o_bx = take((size_t)R * N * 3 * 8),
	             o_pa = take((size_t)R * N * 2 * 4), o_ent = take(params->rescore_entities ? (size_t)R * P * 3 * 4 : 0),
	             o_en = take((size_t)R * 8), o_ord = take((size_t)R * 4), o_cl = take((size_t)R * sizeof(adgpu_cluster)),
	             o_nc = take(4);
	// clustering: the pairs' RMSDs and rows, or the centres and their RMSDs
	const bool by_pairs = R <= kPairRuns;
	const int W = (R + 31) / 32;
	const size_t o_cen = take(by_pairs ? (size_t)R * R * 4 : (size_t)R * 4),
	             o_cr = take(by_pairs ? (size_t)R * W * 4 : (size_t)R * 8);

	unsigned char* d = nullptr;
	auto done = [&](cudaError_t err, const char* what) {
		if (d) cudaFreeAsync(d, st);
		cudaStreamSynchronize(st);
		return err == cudaSuccess ? ADGPU_OK : cuda_fail(err, what);
	};
	cudaError_t e = pool ? cudaMallocFromPoolAsync(reinterpret_cast<void**>(&d), off, pool, st)
	                     : cudaMallocAsync(reinterpret_cast<void**>(&d), off, st);
	if (e != cudaSuccess) { d = nullptr; return done(e, "result scratch"); }
	e = cudaMemcpyAsync(d, blob.data(), blob.size(), cudaMemcpyHostToDevice, st);
	if (e != cudaSuccess) return done(e, "result tables");

	PostDev D;
	memset(&D, 0, sizeof(D));
	D.N = N; D.NL = L.true_lig_atoms; D.NR = NR; D.NT = NT; D.Q = Q; D.P = P;
	D.gx = dp.gridsize_x; D.gy = dp.gridsize_y; D.gz = dp.gridsize_z; D.nmaps = dp.num_of_map_atypes;
	D.rmsd_atoms = L.true_lig_atoms ? L.true_lig_atoms : N;
	D.symmetry = params->handle_symmetry ? 1 : 0;
	D.rescore_all = params->rescore_entities ? 1 : 0;
	D.cells = grid_cells ? 1 : 0;
	D.grid = grid;
	D.ref_xyz = (const double*)(d + o_ref); D.input_xyz = (const double*)(d + o_in); D.charge = (const double*)(d + o_q);
	D.rot_move = (const double*)(d + o_mv); D.rot_unit = (const double*)(d + o_un);
	D.flex_or_cg = flex_or_cg ? 1 : 0;
	D.rot_mask = (const unsigned long long*)(d + o_mask);
	D.rtab = (const float4*)(d + o_rt); D.etab = (const float2*)(d + o_et);
	D.type = (const int*)(d + o_ty); D.map = (const int*)(d + o_map);
	D.ignore = d + o_ig; D.pairs = (const PostPair*)(d + o_pr);
	// get_movvec_to_origo of the reference orientation (host/src/processligand.cpp:1363-1387)
	if (L.true_lig_atoms > 0) {
		double t[3] = {0, 0, 0};
		for (int i = 0; i < L.true_lig_atoms; i++) for (int k = 0; k < 3; k++) t[k] += L.ref_xyz[3 * i + k];
		for (int k = 0; k < 3; k++) D.movvec[k] = -1 * t[k] / L.true_lig_atoms;
	}
	D.spacing = L.spacing;
	for (int k = 0; k < 3; k++) D.origin[k] = L.origin[k];
	D.smooth = dp.smooth;
	D.elec_min_distance = dp.elec_min_distance;

	RunRec* d_runs = (RunRec*)(d + o_runs);
	double* d_bx = (double*)(d + o_bx);
	float* d_pa = (float*)(d + o_pa);
	float* d_ent = params->rescore_entities ? (float*)(d + o_ent) : nullptr;
	adgpu_cluster* d_cl = (adgpu_cluster*)(d + o_cl);
	int* d_nc = (int*)(d + o_nc);

	if (reinterpret_cast<uintptr_t>(populations) % sizeof(float4) == 0)
		arrange_kernel<float4><<<R, 256, (size_t)P * 8, st>>>(populations, energies, (float*)(d + o_scr), P);
	else
		arrange_kernel<float><<<R, 256, (size_t)P * 8, st>>>(populations, energies, (float*)(d + o_scr), P);
	const int ntask = params->rescore_entities ? R * P : R;
	static_assert(kWarps * rescore_warp_bytes(ADGPU_MAX_ATOMS, ADGPU_MAX_ROTBONDS) <= 48 * 1024, "no raised limit needed");
	const size_t wsm = (size_t)kWarps * rescore_warp_bytes(N, NR);
	int dev = 0, sms = 148;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	const int blocks = std::min((ntask + kWarps - 1) / kWarps, sms * 8);
	rescore_kernel<<<blocks, kWarps * 32, wsm, st>>>(D, populations, energies, ntask, d_runs, d_bx, d_pa, d_ent);
	const int free_roaming = params->free_roaming_ligand ? 1 : 0;
	const double tol = (double)params->rmsd_tolerance, torsional = params->coeff_tors * L.true_lig_rotbonds;
	int* d_ord = (int*)(d + o_ord);
	order_kernel<<<1, 1024, 0, st>>>(R, d_runs, (double*)(d + o_en), d_ord, free_roaming);
	if (!params->calc_clustering) {
		e = cudaMemsetAsync(d_nc, 0, 4, st);
	} else if (by_pairs) {
		float* mat = (float*)(d + o_cen);
		unsigned int* bits = (unsigned int*)(d + o_cr);
		const int npair = R * (R - 1) / 2;
		e = cudaMemsetAsync(bits, 0, (size_t)R * W * 4, st);
		if (npair > 0)
			pair_rmsd_kernel<<<std::min((npair + kWarps - 1) / kWarps, sms * 16), kWarps * 32, (size_t)kWarps * N * 8, st>>>(
			    D, R, d_bx, d_ord, tol, mat, bits);
		const size_t rows = (size_t)R * W * 4;
		if (e == cudaSuccess && rows > 40 * 1024) e = allow_smem(cluster_scan_kernel, (size_t)kPairRuns * kPairRuns / 8);
		if (e == cudaSuccess)
			cluster_scan_kernel<<<1, 256, rows, st>>>(R, d_runs, d_ord, mat, bits, params->nr_cluster_poses, free_roaming,
			                                          torsional, d_cl, d_nc);
	} else {
		const size_t csm = (size_t)32 * N * 8;
		if (csm > 48 * 1024) e = allow_smem(cluster_kernel, (size_t)32 * ADGPU_MAX_ATOMS * 8);
		if (e == cudaSuccess)
			cluster_kernel<<<1, 1024, csm, st>>>(D, R, d_runs, d_bx, d_ord, (int*)(d + o_cen), (double*)(d + o_cr), tol,
			                                     params->nr_cluster_poses, free_roaming, torsional, d_cl, d_nc);
	}
	if (e != cudaSuccess) return done(e, "result clustering");
	e = cudaGetLastError();
	if (e != cudaSuccess) return done(e, "result kernels");
	std::vector<RunRec> h_runs(R);
	e = cudaMemcpyAsync(h_runs.data(), d_runs, R * sizeof(RunRec), cudaMemcpyDeviceToHost, st);
	if (e == cudaSuccess) e = cudaMemcpyAsync(clusters_out, d_cl, R * sizeof(adgpu_cluster), cudaMemcpyDeviceToHost, st);
	if (e == cudaSuccess) e = cudaMemcpyAsync(num_clusters, d_nc, 4, cudaMemcpyDeviceToHost, st);
	if (e == cudaSuccess && best_xyz) e = cudaMemcpyAsync(best_xyz, d_bx, (size_t)R * N * 3 * 8, cudaMemcpyDeviceToHost, st);
	if (e == cudaSuccess && peratom) e = cudaMemcpyAsync(peratom, d_pa, (size_t)R * N * 2 * 4, cudaMemcpyDeviceToHost, st);
	if (e == cudaSuccess && entities) e = cudaMemcpyAsync(entities, d_ent, (size_t)R * P * 3 * 4, cudaMemcpyDeviceToHost, st);
	if (e == cudaSuccess) e = cudaStreamSynchronize(st);
	if (e != cudaSuccess) return done(e, "result download");
	for (int r = 0; r < R; r++) {
		const RunRec& s = h_runs[r];
		adgpu_run_result& o = runs_out[r];
		o.inter_e = s.inter; o.interflex_e = s.interflex; o.inter_e_elec = s.elec; o.intra_e = s.intra;
		o.intraflex_e = s.intraflex; o.rmsd_from_ref = s.rmsd; o.rmsd_from_cluster_center = s.crmsd; o.energy = s.energy;
		o.run_number = r + 1; o.cluster_id = s.clus; o.cluster_subrank = s.subrank; o.output = s.output;
		o.energy_rank = s.rank;
	}
	return done(cudaSuccess, "");
}


}  // namespace adgpu

extern "C" {

adgpu_status adgpu_process_result(const adgpu_ligand* lig, const float* grid_reference_layout, float* populations,
                                  float* energies, uint32_t num_runs, const adgpu_result_params* params,
                                  adgpu_run_result* runs_out, adgpu_cluster* clusters_out, int* num_clusters,
                                  double* best_xyz, float* peratom, float* entities)
{
	adgpu::NvtxRange nvtx_range("adgpu_process_result");
	if (!lig) return fail(ADGPU_ERR_ARG, "null argument");
	// a blocking stream: ordered after the caller's work on the legacy
	// default stream (where the kernel API and torch's default stream write
	// the final populations)
	cudaStream_t st = nullptr;
	cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamDefault);
	if (e != cudaSuccess) return cuda_fail(e, "stream");
	// scratch from a pool of this library that keeps its memory between calls
	// (one per device), so repeated calls do not go back to the driver
	static std::mutex pool_mu;
	static cudaMemPool_t pools[64] = {};
	cudaMemPool_t pool = nullptr;
	int dev = 0;
	if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
		std::lock_guard<std::mutex> lk(pool_mu);
		if (!pools[dev]) {
			cudaMemPoolProps props{};
			props.allocType = cudaMemAllocationTypePinned;
			props.location.type = cudaMemLocationTypeDevice;
			props.location.id = dev;
			if (cudaMemPoolCreate(&pools[dev], &props) == cudaSuccess) {
				uint64_t keep = 256ull << 20;
				cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
			} else {
				pools[dev] = nullptr;
				cudaGetLastError();
			}
		}
		pool = pools[dev];
	}
	adgpu_status rc = process_result_core(lig->p.post, lig->p.pairs.data(), lig->p.dockpars, grid_reference_layout, 0,
	                                      populations, energies, num_runs, params, runs_out, clusters_out, num_clusters,
	                                      best_xyz, peratom, entities, st, pool);
	cudaStreamDestroy(st);
	return rc;
}

}  // extern "C"
