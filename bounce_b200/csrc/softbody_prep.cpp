// Soft body preparation on the host.  The element matrices follow the
// reference constructor's float arithmetic step for step (compiled without
// FMA contraction), so the device step starts from bit-identical data:
//   lumped mass rho V / 4 per vertex in element order   softbody.cpp:640-680
//   invE = (e1 e2 e3)^-1 by the adjugate                softbody.cpp:511-520, common/math/math.cpp:111-133
//   D (isotropic elasticity)                            softbody.cpp:43-75
#include "softbody_prep.h"

#include <cmath>
#include <cstring>

#include "../../include/b3g.h"

namespace b3g {

namespace {

struct V3 {
    float x, y, z;
};
inline V3 sub(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
inline float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
inline V3 cross(V3 a, V3 b) { return V3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }

// b3Volume with b3Sign (include/bounce/common/math/vec3.h:226-233, math.h:80-83)
float tet_volume(V3 a, V3 b, V3 c, V3 d)
{
    const float v = dot(sub(b, a), cross(sub(c, a), sub(d, a)));
    const float sign = (float)(0.0f < v) - (float)(v < 0.0f);
    const float inv6 = 1.0f / 6.0f;
    return sign * inv6 * v;
}

// the inverse of the edge matrix (columns e1, e2, e3) by the adjugate, and the volume
void element_shape(V3 p1, V3 p2, V3 p3, V3 p4, float* shape)
{
    const V3 e1 = sub(p2, p1), e2 = sub(p3, p1), e3 = sub(p4, p1);
    // rows of adj are the cross products
    float det = dot(e1, cross(e2, e3));
    if (det != 0.0f) det = 1.0f / det;
    const V3 c1 = cross(e2, e3), c2 = cross(e3, e1), c3 = cross(e1, e2);
    // column-major 3x3: inv[r + 3 c]; adjugate column c holds (c1[c], c2[c], c3[c])
    const float adj[9] = {c1.x, c2.x, c3.x, c1.y, c2.y, c3.y, c1.z, c2.z, c3.z};
    for (int k = 0; k < 9; ++k) shape[k] = det * adj[k];
    shape[9] = tet_volume(p1, p2, p3, p4);
    shape[10] = shape[11] = 0.0f;
}

}  // namespace

int prepare_softbody(uint32_t n, const float* vertices, uint32_t t, const uint32_t* tets, float density, float E,
                     float nu, SoftBodyPrep* out)
{
    SoftBodyPrep& S = *out;
    S = SoftBodyPrep();
    S.n = n;
    S.t = t;
    auto vert = [&](uint32_t i) { return V3{vertices[3 * i], vertices[3 * i + 1], vertices[3 * i + 2]}; };
    for (uint64_t k = 0; k < 4ull * t; ++k)
        if (tets[k] >= n) return B3G_ERR_DEGENERATE_MESH;
    S.mass.assign(n, 0.0f);
    S.shape.resize(12 * (size_t)t);
    S.lambda = (nu * E) / ((1 + nu) * (1 - 2 * nu));
    S.mu = E / (2 * (1 + nu));
    S.lambda2mu = S.lambda + 2 * S.mu;
    const float inv4 = 1.0f / 4.0f;
    for (uint32_t e = 0; e < t; ++e) {
        const uint32_t* tv = tets + 4 * (size_t)e;
        if (tv[0] == tv[1] || tv[0] == tv[2] || tv[0] == tv[3] || tv[1] == tv[2] || tv[1] == tv[3] || tv[2] == tv[3])
            return B3G_ERR_DEGENERATE_MESH;
        const float vol = tet_volume(vert(tv[0]), vert(tv[1]), vert(tv[2]), vert(tv[3]));
        if (!(vol > 0.0f) || !std::isfinite(vol)) return B3G_ERR_DEGENERATE_MESH;
        const float mass = density * vol;
        for (int k = 0; k < 4; ++k) S.mass[tv[k]] += inv4 * mass;
        element_shape(vert(tv[0]), vert(tv[1]), vert(tv[2]), vert(tv[3]), &S.shape[12 * (size_t)e]);
    }
    for (uint32_t i = 0; i < n; ++i)
        if (!(S.mass[i] > 0.0f)) return B3G_ERR_DEGENERATE_MESH;  // a vertex no element uses
    // incidence in element order
    std::vector<uint32_t> cnt(n + 1, 0);
    for (uint64_t k = 0; k < 4ull * t; ++k) ++cnt[tets[k] + 1];
    S.inc_ptr.assign(n + 1, 0);
    for (uint32_t i = 0; i < n; ++i) S.inc_ptr[i + 1] = S.inc_ptr[i] + cnt[i + 1];
    S.inc_elem.resize(4 * (size_t)t);
    S.inc_meta.resize(4 * (size_t)t);
    std::vector<uint32_t> fill(S.inc_ptr.begin(), S.inc_ptr.end() - 1);
    for (uint32_t e = 0; e < t; ++e)
        for (uint32_t k = 0; k < 4; ++k) {
            const uint32_t i = tets[4 * (size_t)e + k];
            S.inc_elem[fill[i]] = e;
            S.inc_meta[fill[i]] = k;
            ++fill[i];
        }
    // block rows in first-touch order, and each incidence's slots
    S.rowptr.assign(n + 1, 0);
    S.diag.assign(n, 0);
    std::vector<uint32_t> row;
    for (uint32_t i = 0; i < n; ++i) {
        row.clear();
        for (uint32_t q = S.inc_ptr[i]; q < S.inc_ptr[i + 1]; ++q) {
            const uint32_t* tv = tets + 4 * (size_t)S.inc_elem[q];
            uint32_t meta = S.inc_meta[q];
            for (uint32_t j = 0; j < 4; ++j) {
                uint32_t slot = 0;
                while (slot < row.size() && row[slot] != tv[j]) ++slot;
                if (slot == row.size()) row.push_back(tv[j]);
                if (slot > 127) return B3G_ERR_UNSUPPORTED;
                meta |= slot << (4 + 7 * j);
            }
            S.inc_meta[q] = meta;
        }
        S.rowptr[i + 1] = S.rowptr[i] + (uint32_t)row.size();
        for (uint32_t k = 0; k < row.size(); ++k) {
            if (row[k] == i) S.diag[i] = S.rowptr[i] + k;
            S.cols.push_back(row[k]);
        }
        if (row.size() > S.max_deg) S.max_deg = (uint32_t)row.size();
    }
    return 0;
}

}  // namespace b3g
