// Test harness for the traversal's slab test (cupbr_b200/csrc/slab.hpp): reads
// n rays (origin, direction: 6 float32 each) from argv[1], the box (centre,
// half extent per axis: 6 float32) from argv[2], writes 3 int32 per ray to
// argv[3]: whether it walks a tree, whether a missing child is accepted,
// whether the box is.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "slab.hpp"

static std::vector<float> read_all(const char* path) {
    std::vector<float> v;
    float x;
    if (FILE* f = std::fopen(path, "rb")) {
        while (std::fread(&x, sizeof x, 1, f) == 1) v.push_back(x);
        std::fclose(f);
    }
    return v;
}

int main(int argc, char** argv) {
    if (argc != 4) return 2;
    const std::vector<float> rays = read_all(argv[1]), b = read_all(argv[2]);
    FILE* o = std::fopen(argv[3], "wb");
    if (!o || b.size() != 6) return 3;
    const float none = -INFINITY;
    for (size_t i = 0; i + 5 < rays.size(); i += 6) {
        const float* r = &rays[i];
        const cupbr_b200::SlabRay s = cupbr_b200::slab_ray(r[0], r[1], r[2], r[3], r[4], r[5]);
        float t;
        const int32_t out[3] = {cupbr_b200::slab_walks(s, r[3], r[4], r[5]),
                                cupbr_b200::slab_child(0.0f, none, 0.0f, none, 0.0f, none, s, INFINITY, t),
                                cupbr_b200::slab_child(b[0], b[1], b[2], b[3], b[4], b[5], s, INFINITY, t)};
        std::fwrite(out, sizeof out, 1, o);
    }
    std::fclose(o);
    return 0;
}
