// Per-cell kernels: seeding, count correction with the new layout,
// projection partial sums and the DoF gather.
//
// Count correction (check_particle_distribution,
// src/pfem2particlehandler.cpp:356-410) depends on per-(cell, part) counts
// only: a part keeps min(count, max+1) particles, here the ones with the
// smallest key(id), and every real part left without particles in a cell
// that had any gets one new particle at its centre.  New ids continue the
// running count in (cell ascending, part x-major) order, the order in which
// the reference hands them out.
//
// Layout after a step: cells in ascending order; inside a cell the particles
// that stayed (in their previous order), then the ones that moved in (by
// key), then the new ones (by part).  Each cell owns `count + new` slots,
// known from the move's per-cell count and part occupancy before the write
// pass starts; a cell whose over-full parts lose particles leaves that many
// empty slots (cell = HOLE) at the end of its range.  The layout and every
// floating-point sum taken over it are deterministic.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "geom32.cuh"
#include "geom64.cuh"
#include "staging.cuh"

namespace pfem2 {

template <typename Real>
__device__ __forceinline__ Real ldr(const void* p, uint32_t i)
{
    return reinterpret_cast<const Real*>(p)[i];
}

template <typename Real>
__device__ __forceinline__ void str(void* p, uint32_t i, Real v)
{
    reinterpret_cast<Real*>(p)[i] = v;
}

// Velocity interpolation at xi from the cell's vertex velocities (FP64 form).
template <int DIM, typename Real>
__device__ __forceinline__ void interp_v(const void* Vc, uint32_t c, const Real* xi, Real* u)
{
    constexpr int NV = 1 << DIM, VS = Dims<DIM>::VS;
    const Real* p = reinterpret_cast<const Real*>(Vc) + (size_t)c * NV * VS;
    Real N[NV];
    if constexpr (std::is_same<Real, double>::value) shape64<DIM>(xi, N);
    else shape32<DIM>(xi, N);
#pragma unroll
    for (int d = 0; d < DIM; ++d) u[d] = Real(0);
#pragma unroll
    for (int iv = 0; iv < NV; ++iv)
#pragma unroll
        for (int d = 0; d < DIM; ++d) u[d] = u[d] + N[iv] * __ldg(p + iv * VS + d);
}

// A new particle at the centre of part idx of cell c (seed_particles
// :87-104 and check_particle_distribution :390-407): xi = (idx + 1/2) h,
// x = F(xi) (FP64 form), v = V interpolated at xi in FP64 (rounded to the
// form's precision).
template <int DIM, typename Real>
__device__ __forceinline__ void new_particle_at(const StepArgs& a, uint32_t c, const int* idx, Real* xi, Real* v,
                                                double* x)
{
    double xid[DIM], vd[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        xid[d] = (idx[d] + 0.5) * a.pp.h[d];
        xi[d] = (Real)xid[d];
    }
    velocity_from_dofs<DIM>(a.mesh.cd, a.Va, c, xid, vd);
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = (Real)vd[d];
    if constexpr (std::is_same<Real, double>::value) {
        double X[1 << DIM][DIM];
        load_cell64<DIM>(a.mesh.cellX, c, X);
        fwd64<DIM>(X, xid, x);
    }
}

// The same stored into slot dst of a state.
template <int DIM, typename Real>
__device__ __forceinline__ void new_particle(const StepArgs& a, const PartState& S, uint32_t dst, uint32_t c,
                                             const int* idx, uint32_t id)
{
    Real xi[DIM], v[DIM];
    double x[DIM];
    new_particle_at<DIM, Real>(a, c, idx, xi, v, x);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        if constexpr (std::is_same<Real, double>::value) str<double>(S.x[d], dst, x[d]);
        str<Real>(S.xi[d], dst, xi[d]);
        str<Real>(S.v[d], dst, v[d]);
    }
    S.cell[dst] = c;
    S.id[dst] = id;
}

template <int DIM>
__device__ __forceinline__ void part_digits(int k, const PartParams& pp, int* idx)
{
    idx[2] = 0;
    if (DIM == 2) {
        idx[0] = k / pp.q[1];
        idx[1] = k % pp.q[1];
    } else {
        idx[0] = k / (pp.q[1] * pp.q[2]);
        idx[1] = (k / pp.q[2]) % pp.q[1];
        idx[2] = k % pp.q[2];
    }
}

// seed_particles (:43-109): npart particles per owned cell, cell-major, parts
// x-major; ids by the global (cell, part) index, so a partitioned run hands
// out the ids of an unpartitioned one.  Cells outside [cbeg, cend) get empty
// ranges.
template <int DIM, typename Real>
__global__ void k_seed(StepArgs a, uint32_t* cell_start)
{
    const uint32_t cb = (uint32_t)a.cbeg, ce = (uint32_t)a.cend;
    const uint32_t total = (ce - cb) * a.pp.npart;
    const uint32_t id0 = a.stats->next_id + cb * a.pp.npart;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t c = cb + t / a.pp.npart;
        const int k = (int)(t % a.pp.npart);
        int idx[3];
        part_digits<DIM>(k, a.pp, idx);
        new_particle<DIM, Real>(a, a.S0, t, c, idx, id0 + t + 1);
        if (k == 0) cell_start[c] = t;
        if (a.chunk_first && t % ADV_REC == 0) a.chunk_first[t / ADV_REC] = c;
    }
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < (uint32_t)a.mesh.nC; c += gridDim.x * blockDim.x)
        if (c < cb || c >= ce) cell_start[c] = c < cb ? 0u : total;
    if (blockIdx.x == 0 && threadIdx.x == 0) cell_start[a.mesh.nC] = total;
}

__device__ __forceinline__ int survivors(int cnt, int maxpp, int apply)
{
    if (!apply) return cnt;
    if (maxpp < 0) return 0;
    return cnt < maxpp + 1 ? cnt : maxpp + 1;
}

// Does extended part p get a new particle?  (A real part with no survivor in
// a cell that had particles.)
__device__ __forceinline__ bool gets_seed(const StepArgs& a, int p, int cnt, uint32_t n)
{
    if (!a.apply_counts || n == 0 || p >= a.pp.npe) return false;
    if (!((a.pp.realmask[p >> 6] >> (p & 63)) & 1ull)) return false;
    return survivors(cnt, a.pp.maxpp, 1) == 0;
}

// ---------------------------------------------------------------------------
// Projection partials: per cell and local vertex iv, sum_p N_iv v_p and
// sum_p N_iv (project_particle_fields :191-199 restricted to one cell), in
// the cell's particle order.  Each lane writes one particle's 4*NV terms as a
// row of a per-warp shared array; lane e then adds column e row by row
// (FP32: Kahan-compensated).  Entry e = iv*4 + comp, comp = DIM is the weight.
// ---------------------------------------------------------------------------

// Row stride of the partial-row array: 36 keeps rows 16-byte aligned (vector
// stores) and the column reads (lane e reads entry e of row r) conflict-free.
constexpr int TRW = 36;

template <typename Real>
struct PartialAcc {
    Real s = Real(0), c = Real(0);
};

template <int DIM, typename Real>
__device__ __forceinline__ void partial_row(Real (*tr)[TRW], int row, const Real* xi, const Real* v)
{
    constexpr int NV = 1 << DIM;
    Real N[NV];
    if constexpr (std::is_same<Real, double>::value) shape64<DIM>(xi, N);
    else shape32<DIM>(xi, N);
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        if constexpr (std::is_same<Real, float>::value) {
            float4 t;
            t.x = N[iv] * v[0];
            t.y = N[iv] * v[1];
            t.z = DIM == 3 ? N[iv] * v[DIM - 1] : N[iv];
            t.w = DIM == 3 ? N[iv] : 0.0f;
            *reinterpret_cast<float4*>(&tr[row][iv * 4]) = t;
        } else {
#pragma unroll
            for (int d = 0; d < DIM; ++d) tr[row][iv * 4 + d] = N[iv] * v[d];
            tr[row][iv * 4 + DIM] = N[iv];
            if (DIM == 2) tr[row][iv * 4 + 3] = 0.0;
        }
    }
}

// Column sums of up to 32 partial rows into acc (lane = column).  FP64:
// the rows in order, as the oracle adds them.  FP32: a pairwise tree over the
// 32 rows (empty rows read as 0), then one compensated add into acc.
template <int DIM, typename Real>
__device__ __forceinline__ void partial_sum_rows(Real (*tr)[TRW], int rows, int lane, PartialAcc<Real>& acc)
{
    constexpr int PW = Dims<DIM>::PW;
    if (lane < PW) {
        if constexpr (std::is_same<Real, double>::value) {
            for (int r = 0; r < rows; ++r) acc.s = acc.s + tr[r][lane];
        } else {
            float t[32];
#pragma unroll
            for (int r = 0; r < 32; ++r) t[r] = r < rows ? tr[r][lane] : 0.0f;
#pragma unroll
            for (int w = 16; w >= 1; w >>= 1)
#pragma unroll
                for (int r = 0; r < w; ++r) t[r] = t[r] + t[r + w];
            const float y = t[0] - acc.c;
            const float s = acc.s + y;
            acc.c = (s - acc.s) - y;
            acc.s = s;
        }
    }
}

template <int DIM, typename Real>
__device__ __forceinline__ void store_partial(const StepArgs& a, uint32_t c, const PartialAcc<Real>& acc, int lane)
{
    constexpr int PW = Dims<DIM>::PW;
    if (lane < PW) reinterpret_cast<Real*>(a.partials)[(size_t)c * PW + lane] = acc.s - acc.c;
}

// Partials of the particles in slots [b, b+count) of a state, in order
// (empty slots contribute nothing).
template <int DIM, typename Real>
__device__ __forceinline__ void partials_of_range(const StepArgs& a, const PartState& S, uint32_t c, uint32_t b,
                                                  uint32_t count, Real (*tr)[TRW], int lane)
{
    PartialAcc<Real> acc;
    for (uint32_t base = 0; base < count; base += 32) {
        const uint32_t j = base + lane;
        const bool valid = j < count && S.cell[b + j] != HOLE;
        Real xi[DIM], v[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            xi[d] = valid ? ldr<Real>(S.xi[d], b + j) : Real(0);
            v[d] = valid ? ldr<Real>(S.v[d], b + j) : Real(0);
        }
        const int rows = count - base < 32 ? (int)(count - base) : 32;
        if (valid) {
            partial_row<DIM, Real>(tr, lane, xi, v);
        } else if (lane < rows) {  // an empty slot adds nothing
#pragma unroll
            for (int k = 0; k < Dims<DIM>::PW; ++k) tr[lane][k] = Real(0);
        }
        __syncwarp();
        partial_sum_rows<DIM, Real>(tr, rows, lane, acc);
        __syncwarp();
    }
    store_partial<DIM, Real>(a, c, acc, lane);
}

// ---------------------------------------------------------------------------

// Partials of the current state (after seeding or an upload).
template <int DIM, typename Real>
__global__ void __launch_bounds__(CELL_WARPS * 32) k_partials(StepArgs a, const uint32_t* cell_start)
{
    __shared__ __align__(16) Real tr_s[CELL_WARPS][32][TRW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = blockIdx.x * CELL_WARPS + warp; c < a.mesh.nC; c += gridDim.x * CELL_WARPS) {
        const uint32_t b = cell_start[c], e = cell_start[c + 1];
        partials_of_range<DIM, Real>(a, a.S0, (uint32_t)c, b, e - b, tr_s[warp], lane);
    }
}

// Standalone velocity correction of the current state (when no move follows).
template <int DIM, typename Real>
__global__ void k_correct(StepArgs a)
{
    const uint32_t n = (uint32_t)a.stats->n_slots;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = a.S0.cell[i];
        if (c >= (uint32_t)a.mesh.nC) continue;
        Real xi[DIM], corr[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) xi[d] = ldr<Real>(a.S0.xi[d], i);
        if constexpr (std::is_same<Real, double>::value) {
            interp_v<DIM, Real>(a.dVc, c, xi, corr);
        } else {
            Rec32<DIM> r;
            load_rec32<DIM>(a.dvrec32, c, r);
            eval_poly<DIM>(r.b, xi, corr);
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) str<Real>(a.S0.v[d], i, ldr<Real>(a.S0.v[d], i) + corr[d]);
    }
}

// The 4 values of one (cell, vertex) partial entry (16-byte aligned).
__device__ __forceinline__ void load4(const float* p, float* q)
{
    const float4 t = __ldg(reinterpret_cast<const float4*>(p));
    q[0] = t.x;
    q[1] = t.y;
    q[2] = t.z;
    q[3] = t.w;
}
__device__ __forceinline__ void load4(const double* p, double* q)
{
    const double2 t0 = __ldg(reinterpret_cast<const double2*>(p));
    const double2 t1 = __ldg(reinterpret_cast<const double2*>(p) + 1);
    q[0] = t0.x;
    q[1] = t0.y;
    q[2] = t1.x;
    q[3] = t1.y;
}

// DoF gather: V_d = sum num_d / sum den over the cells sharing the DoF, in
// ascending cell order, FP64 sums and division (0/0 -> NaN as the reference,
// or the kept input value under empty_dof_policy 1).  Up to 8 cell entries
// are fetched before any is summed; a thread's first DoF's entries (mesh
// data) are fetched before the kernel waits for the write pass.
template <int DIM, typename PReal>
__global__ void k_gather(StepArgs a, int keep_empty)
{
    constexpr int NV = 1 << DIM, PW = Dims<DIM>::PW;
    const int stride = gridDim.x * blockDim.x;
    const int nloop = (a.mesh.nD + stride - 1) / stride * stride;
    const int dof0 = blockIdx.x * blockDim.x + threadIdx.x;
    int32_t b0 = 0, e0 = 0, ent0[8];
    if (dof0 < a.mesh.nD) {
        b0 = __ldg(a.mesh.d2c_off + dof0);
        e0 = __ldg(a.mesh.d2c_off + dof0 + 1);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ent0[j] = b0 + j < e0 ? __ldg(a.mesh.d2c_ent + b0 + j) : -1;
    pdl_entry();
    const PReal* P = reinterpret_cast<const PReal*>(a.partials);
    unsigned long long nan_dofs = 0;
    for (int dof = dof0; dof < nloop; dof += stride) {
        if (dof >= a.mesh.nD) continue;
        double num[DIM], den = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) num[d] = 0.0;
        const bool first = dof == dof0;
        const int32_t b = first ? b0 : __ldg(a.mesh.d2c_off + dof), e = first ? e0 : __ldg(a.mesh.d2c_off + dof + 1);
        for (int32_t k0 = b; k0 < e; k0 += 8) {
            int32_t ent[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                ent[j] = first && k0 == b ? ent0[j] : k0 + j < e ? __ldg(a.mesh.d2c_ent + k0 + j) : -1;
            PReal q[8][4];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int32_t en = ent[j] < 0 ? 0 : ent[j];
                load4(P + (size_t)(en / NV) * PW + (en % NV) * 4, q[j]);  // one vector load per entry
                if (ent[j] < 0) q[j][0] = q[j][1] = q[j][2] = q[j][3] = PReal(0);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (ent[j] < 0) continue;
#pragma unroll
                for (int d = 0; d < DIM; ++d) num[d] = num[d] + (double)q[j][d];
                den = den + (double)q[j][DIM];
            }
        }
        if (den == 0.0) nan_dofs++;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            double r = num[d] / den;
            if (den == 0.0 && keep_empty) r = a.Vkeep[(size_t)d * a.mesh.nD + dof];
            a.Vout[(size_t)d * a.mesh.nD + dof] = r;
            if (a.Vout2) a.Vout2[(size_t)d * a.mesh.nD + dof] = r;
        }
    }
    nan_dofs = warp_sum_u64(nan_dofs);
    if ((threadIdx.x & 31) == 0 && nan_dofs) atomicAdd(&a.stats->nan_dofs, nan_dofs);
}

// Global positions of the FP32 form for output: x = F(xi) in FP64.
template <int DIM>
__global__ void k_positions32(StepArgs a, double* xout)
{
    const uint32_t n = (uint32_t)a.stats->n_slots;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = a.S0.cell[i];
        double X[1 << DIM][DIM], xi[DIM], x[DIM];
        if (c >= (uint32_t)a.mesh.nC) continue;
        load_cell64<DIM>(a.mesh.cellX, c, X);
#pragma unroll
        for (int d = 0; d < DIM; ++d) xi[d] = (double)ldr<float>(a.S0.xi[d], i);
        fwd64<DIM>(X, xi, x);
#pragma unroll
        for (int d = 0; d < DIM; ++d) xout[(size_t)i * DIM + d] = x[d];
    }
}

// Output packing (output_particle_solution, src/pfem2particlehandler.cpp:
// 218-317, writes positions and velocities as Float32): for the k-th live
// particle (slot[k], in slot order) out[3k..3k+2] = x and
// out[3n + 3k..] = v as floats, x = the FP64 position (FP64 form) or F(xi)
// in FP64 (FP32 form); 2D pads the third component with 0.
template <int DIM, typename Real>
__global__ void k_pack_output(StepArgs a, const uint32_t* __restrict__ slot, uint32_t n, float* __restrict__ out)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t i = slot[k];
        double x[3] = {0.0, 0.0, 0.0};
        if constexpr (std::is_same<Real, double>::value) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) x[d] = ldr<double>(a.S0.x[d], i);
        } else {
            double X[1 << DIM][DIM], xi[DIM];
            load_cell64<DIM>(a.mesh.cellX, a.S0.cell[i], X);
#pragma unroll
            for (int d = 0; d < DIM; ++d) xi[d] = (double)ldr<float>(a.S0.xi[d], i);
            fwd64<DIM>(X, xi, x);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            out[(size_t)3 * k + d] = (float)x[d];
            out[(size_t)3 * n + (size_t)3 * k + d] = d < DIM ? (float)ldr<Real>(a.S0.v[d], i) : 0.0f;
        }
    }
}

}  // namespace pfem2
