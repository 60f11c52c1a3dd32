// tg_consumers.cu -- algorithm kernels that read resident relations in place
// through include/tetragpu_device.h, as a caller's own kernels would (the
// reference's aim for its relation kernels, src/cuda_extraction.cu:16-22).
//
//   tg_get_device_mesh  every resident relation's device pointers
//   tg_smooth_field     Laplacian smoothing of a vertex field over VV: each
//                       step replaces f[v] by the mean of f[v] and its
//                       neighbours' values (ping-pong between two buffers)
#include <algorithm>

#include "tetragpu.h"
#include "tetragpu_device.h"
#include "tg_internal.h"

namespace tg {
namespace {

__global__ void __launch_bounds__(256)
k_smooth(tg_device_mesh m, const float *__restrict__ in, float *__restrict__ out)
{
    griddep_wait();
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= m.n_verts) return;
    const int32_t n = tg_row_size(m.vv, v);
    const int32_t *nb = tg_row(m.vv, v);
    float s = in[v];
    for (int32_t i = 0; i < n; i++) s += in[nb[i]];
    out[v] = s / (float)(n + 1);
}

// The same over VV by position (rows of positions, padded with -1 to whole
// sectors; values by position): a block's values lie together.  order: scatter
// the result to the vertices (the last step), or null.
__global__ void __launch_bounds__(256)
k_smooth_ordered(const int64_t *__restrict__ off, const int *__restrict__ ent, int64_t V,
                 const float *__restrict__ in, const int *__restrict__ order, float *__restrict__ out)
{
    griddep_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    const int64_t b = off[i];
    const int words = (int)(off[i + 1] - b);
    float s = in[i];
    int n = 0;
    for (int k = 0; k < words; k += 8) {
        unsigned u[8];
        load8(reinterpret_cast<const unsigned *>(ent + b + k), u);
#pragma unroll
        for (int t = 0; t < 8; t++)
            if ((int)u[t] >= 0) {
                s += in[u[t]];
                n++;
            }
    }
    out[order ? order[i] : i] = s / (float)(n + 1);
}

// From this many vertices and steps on the steps run over VV by position.  A
// step by id gathers the neighbours' values from a line each: 16.7 us on 64^3
// cubes (0.27 M vertices, ids permuted) against 2.6 by position, 113 against 32
// on 128^3.  Making the rows costs 45 us on 64^3 and 190 on 128^3, kept on the
// mesh like VV; a first call of five steps, them included: 94 us against 114 on
// 64^3, 433 against 604 on 128^3, but 74 against 72 on 48^3 (0.12 M), where
// both kinds of step are bound by their launches.
constexpr int64_t kOrderVerts = 1 << 17;
static_assert(kOrderVerts >= kOrderField, "whether ids are as good is known from there on");
// The vertices, the steps and the mesh's order alone decide, so that a call gives
// the same bits whether or not the mesh has those rows already.  Meshes whose
// link graph is in the order of ids stay by id (lg_by_id, tg_api.cu): ten steps
// by id and by position, ids in order: 54 and 50 us on 64^3, 311 and 348 on
// 128^3; cells scattered: 54 and 116 on 64^3, with ids permuted too 175 and 117.
constexpr int kOrderSteps = 5;

}  // namespace
}  // namespace tg

using namespace tg;

extern "C" tg_status tg_get_device_mesh(const tg_mesh *mesh, tg_device_mesh *out)
{
    if (!mesh || !out) {
        set_last_error("NULL argument");
        return TG_ERR_INVALID_ARGUMENT;
    }
    tg_device_mesh m{};
    tg_mesh_counts(mesh, &m.n_verts, &m.n_edges, &m.n_faces, &m.n_cells);
    tg_get_tv(mesh, &m.tv);
    auto fixed = [&](int r, tg_fixed_view &v) {
        const int64_t *off;
        const int32_t *ent;
        int64_t rows, n;
        int32_t w;
        if (tg_get_relation(mesh, r, &off, &ent, &rows, &n, &w) == TG_OK) v = {ent, rows, w};
    };
    auto csr = [&](int r, tg_csr_view &v) {
        const int64_t *off;
        const int32_t *ent;
        int64_t rows, n;
        int32_t w;
        if (tg_get_relation(mesh, r, &off, &ent, &rows, &n, &w) == TG_OK) v = {off, ent, rows};
    };
    fixed(TG_REL_TE, m.te);
    fixed(TG_REL_EV, m.ev);
    fixed(TG_REL_TF, m.tf);
    fixed(TG_REL_FV, m.fv);
    fixed(TG_REL_FE, m.fe);
    fixed(TG_REL_FT, m.ft);
    csr(TG_REL_ET, m.et);
    csr(TG_REL_EF, m.ef);
    csr(TG_REL_VT, m.vt);
    csr(TG_REL_TT, m.tt);
    csr(TG_REL_FF, m.ff);
    csr(TG_REL_EE, m.ee);
    csr(TG_REL_VV, m.vv);
    set_last_error("");   // relations not extracted are NULL, not an error
    *out = m;
    return TG_OK;
}

extern "C" tg_status tg_smooth_field(tg_mesh *mesh, const float *in, float *out, int iterations,
                                     float *scratch, void *stream)
{
    if (!mesh || !in || !out || iterations < 0 || (iterations > 1 && !scratch)) {
        set_last_error("NULL argument, negative iterations, or no scratch for more than one");
        return TG_ERR_INVALID_ARGUMENT;
    }
    cudaStream_t s = (cudaStream_t)stream;
    tg_status st = tg_extract(mesh, TG_VV, 0, stream);   // no-op when VV is resident
    if (st != TG_OK) return st;
    tg_device_mesh m;
    tg_get_device_mesh(mesh, &m);
    const unsigned grid = (unsigned)std::max<int64_t>((m.n_verts + 255) / 256, 1);
    if (iterations == 0) {
        if (cudaMemcpyAsync(out, in, (size_t)m.n_verts * 4, cudaMemcpyDeviceToDevice, s) !=
            cudaSuccess) {
            (void)cudaGetLastError();
            set_last_error("cudaMemcpyAsync failed");
            return TG_ERR_CUDA;
        }
        return TG_OK;
    }
    // (under capture the steps are recorded by id: nothing is made then)
    if (m.n_verts >= kOrderVerts && iterations >= kOrderSteps && !capturing(s)) {
        LinkGraph g{};
        // without the memory for them: by id
        if (link_rows(mesh, s, &g) == TG_OK && g.off) {
            // steps alternate between the two buffers so that the last one
            // reads scratch
            float *src = iterations % 2 ? scratch : out, *dst = iterations % 2 ? out : scratch;
            launch_field_in_order(in, g.order, m.n_verts, src, s);
            for (int k = 0; k < iterations; k++) {
                const bool last = k == iterations - 1;
                Launch L("k_smooth_ordered", s);
                launch_pdl(k_smooth_ordered, grid, 256, 0, s, g.off, g.ent, m.n_verts,
                           (const float *)src, last ? g.order : nullptr, last ? out : dst);
                std::swap(src, dst);
            }
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) {
                set_last_error(cudaGetErrorString(e));
                return TG_ERR_CUDA;
            }
            return note_reader(mesh, s, true);
        }
    }
    // steps alternate between out and scratch so that the last one lands in out
    const float *src = in;
    for (int k = 0; k < iterations; k++) {
        float *dst = ((iterations - 1 - k) % 2 == 0) ? out : scratch;
        if (m.n_verts > 0) {
            Launch L("k_smooth", s);
            launch_pdl(k_smooth, grid, 256, 0, s, m, src, dst);
        }
        src = dst;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_last_error(cudaGetErrorString(e));
        return TG_ERR_CUDA;
    }
    return note_reader(mesh, s, false);
}
