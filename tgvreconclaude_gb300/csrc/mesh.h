// A surface mesh: in its context's output buffers on the device, or in host memory.
//
// Host code without the CUDA headers: the device copy is the caller's (surface.cu),
// so the states that a failed copy or allocation leaves can be tested on the CPU.
#pragma once
#include <stdint.h>

#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <utility>

#include "tgvg.h"

struct CUstream_st;

// The mesh whose data is in a context's surface output buffers (surface.cu),
// shared by the context and the mesh; mu orders reads, moves to the host and frees.
struct tgvg_mesh_link {
    std::mutex mu;
    tgvg_mesh* held = nullptr;
    CUstream_st* stream = nullptr;
};

// A mesh stays in the context's own output buffers (B_S_VERTS, B_S_FACES,
// B_S_NRM, which the context keeps between calls anyway) until something else
// needs them, so a read is one copy from the device straight into the caller's
// arrays.  The next extraction, tgvg_compute_normals or tgvg_destroy first moves
// it to host memory: no more than one mesh per context is on the device, and a
// mesh can be read at any time, from any thread, also after the context is gone.
// (Copying every mesh to host vectors and from there to the caller took 16 of
// the 20 ms of a 1.9 M-cube extraction: zero filling the vectors, page faults
// and a single-threaded copy of 150 MB; now 0.9 ms.)
struct tgvg_mesh {
    int64_t nv = 0, nf = 0;       // vertices, triangles
    bool has_normals = false;
    std::shared_ptr<tgvg_mesh_link> link;  // set while the mesh may be on the device
    const float* d_verts = nullptr;        // 3 per vertex
    const uint32_t* d_faces = nullptr;     // 3 per triangle
    const float* d_normals = nullptr;      // 3 per vertex
    std::unique_ptr<float[]> verts;        // the same in host memory, once moved there whole
    std::unique_ptr<uint32_t[]> faces;
    std::unique_ptr<float[]> normals;
    int lost = TGVG_OK;           // why it could not be moved when its context went
};

namespace tgvg {

// Moves the mesh that is on the device, if any, to host memory.  copy(m, v, f, n)
// brings m's arrays to host ones and returns a TGVG code.  The mesh changes only
// when all of it has arrived: after an error it is on the device as before.
template <class Copy>
int mesh_to_host(tgvg_mesh_link* l, Copy copy) {
    std::lock_guard<std::mutex> lk(l->mu);
    tgvg_mesh* m = l->held;
    if (!m) return TGVG_OK;
    std::unique_ptr<float[]> v(new (std::nothrow) float[3 * m->nv + 1]), n;
    std::unique_ptr<uint32_t[]> f(new (std::nothrow) uint32_t[3 * m->nf + 1]);
    if (m->has_normals) n.reset(new (std::nothrow) float[3 * m->nv + 1]);
    if (!v || !f || (m->has_normals && !n)) return TGVG_ERR_NOMEM;
    const int rc = copy(m, v.get(), f.get(), n.get());
    if (rc) return rc;
    m->verts = std::move(v);
    m->faces = std::move(f);
    m->normals = std::move(n);
    m->d_verts = m->d_normals = nullptr;
    m->d_faces = nullptr;
    l->held = nullptr;
    return TGVG_OK;
}

// The context goes: a mesh that cannot be moved is lost, and says so when read.
template <class Copy>
void mesh_release(tgvg_mesh_link* l, Copy copy) {
    const int rc = mesh_to_host(l, copy);
    std::lock_guard<std::mutex> lk(l->mu);
    if (l->held) l->held->lost = rc;
    l->held = nullptr;
}

// Copies the mesh out (null: not wanted) from where it is.
template <class Copy>
int mesh_read(const tgvg_mesh* m, float* v, uint32_t* f, float* n, Copy copy) {
    if (m->link) {
        std::lock_guard<std::mutex> lk(m->link->mu);
        if (m->link->held == m) return copy(m, v, f, n);
        if (m->lost) return m->lost;
    }
    if (v && m->verts) std::memcpy(v, m->verts.get(), 12ull * m->nv);
    if (f && m->faces) std::memcpy(f, m->faces.get(), 12ull * m->nf);
    if (n && m->normals) std::memcpy(n, m->normals.get(), 12ull * m->nv);
    return TGVG_OK;
}

}  // namespace tgvg
