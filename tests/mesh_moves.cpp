// Moves of a mesh to host memory that fail (csrc/mesh.h), with stubs for the
// device copy and for the host's memory.  Exits 0 when every state is as it should be.
#include <cstdio>

#include "mesh.h"

static int fail_alloc = -1;  // the allocation that fails, counted down; -1: none
void* operator new[](std::size_t n, const std::nothrow_t&) noexcept {
    if (fail_alloc >= 0 && fail_alloc-- == 0) return nullptr;
    return ::operator new[](n);
}

static const float DV[3] = {1, 2, 3}, DN[3] = {0, 0, 1};
static const uint32_t DF[6] = {0, 0, 0, 0, 0, 0};
static int copy_rc = TGVG_OK;
static int copy(const tgvg_mesh* m, float* v, uint32_t* f, float* n) {
    if (copy_rc) return copy_rc;
    if (v) std::memcpy(v, m->d_verts, 12 * m->nv);
    if (f) std::memcpy(f, m->d_faces, 12 * m->nf);
    if (n && m->has_normals) std::memcpy(n, m->d_normals, 12 * m->nv);
    return TGVG_OK;
}

static std::unique_ptr<tgvg_mesh> on_device(const std::shared_ptr<tgvg_mesh_link>& l) {
    auto m = std::make_unique<tgvg_mesh>();
    m->nv = 1; m->nf = 2; m->has_normals = true;
    m->d_verts = DV; m->d_faces = DF; m->d_normals = DN;
    m->link = l;
    l->held = m.get();
    return m;
}
// The whole mesh, or `rc` and the caller's arrays untouched.
static bool reads(const tgvg_mesh* m, int rc) {
    float v[3] = {9, 9, 9}, n[3] = {9, 9, 9};
    uint32_t f[6] = {9, 9, 9, 9, 9, 9};
    if (tgvg::mesh_read(m, v, f, n, copy) != rc) return false;
    return rc ? v[0] == 9 && f[0] == 9 && n[0] == 9 : !std::memcmp(v, DV, 12) && !std::memcmp(f, DF, 24) && !std::memcmp(n, DN, 12);
}

int main() {
    int bad = 0;
    auto want = [&](bool ok, const char* what, int k) {
        if (!ok) { std::printf("%s (%d)\n", what, k); ++bad; }
    };
    for (int k = -2; k < 3; ++k) {  // -2: nothing fails, -1: the copy, 0..2: an allocation
        const int rc = k == -2 ? TGVG_OK : k == -1 ? TGVG_ERR_CUDA : TGVG_ERR_NOMEM;
        auto set = [&] { copy_rc = k == -1 ? TGVG_ERR_CUDA : TGVG_OK; fail_alloc = k >= 0 ? k : -1; };
        auto clear = [&] { copy_rc = TGVG_OK; fail_alloc = -1; };
        {  // another extraction wants the buffers
            auto l = std::make_shared<tgvg_mesh_link>();
            auto m = on_device(l);
            set();
            want(tgvg::mesh_to_host(l.get(), copy) == rc, "move's code", k);
            clear();
            want((l->held == m.get()) == (rc != TGVG_OK), "still held after a failed move only", k);
            want(reads(m.get(), TGVG_OK), "readable after the move", k);
            want(tgvg::mesh_to_host(l.get(), copy) == TGVG_OK && !l->held && reads(m.get(), TGVG_OK), "moved again", k);
        }
        {  // the context goes
            auto l = std::make_shared<tgvg_mesh_link>();
            auto m = on_device(l);
            set();
            tgvg::mesh_release(l.get(), copy);
            clear();
            want(!l->held, "not held", k);
            want(reads(m.get(), rc), "read after the context", k);
        }
    }
    return bad != 0;
}
