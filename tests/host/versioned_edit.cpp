// Parameter edits beside running jobs (rebind_parameters_versioned) with each of
// their allocations failing in turn: a rejected edit leaves the scene as it
// was, a later one takes effect.
#include "fake_cuda.h"

#include <cstdio>

#define CHECK(x)                                              \
    do {                                                      \
        if (!(x)) {                                           \
            std::printf("line %d: %s\n", __LINE__, #x);       \
            return 1;                                         \
        }                                                     \
    } while (0)

int main() {
    psy_context *context = nullptr;
    CHECK(psy_context_create(0, &context) == PSY_OK);
    const float positions[9] = {0, 0, 0, 1, 0, 0, 0, 1, 0};
    const uint32_t indices[3] = {0, 1, 2};
    psy_mesh_desc mesh{};
    mesh.positions = positions;
    mesh.indices = indices;
    mesh.vertex_count = 3;
    mesh.triangle_count = 1;
    psy_instance_desc instance{};
    for (int k = 0; k < 4; ++k) instance.object_to_world[5 * k] = 1.0f;
    instance.visibility = PSY_VISIBILITY_ALL;
    // one emissive material: colour in the vector block, strength in the scalars
    psy_closure_instruction closure{};
    closure.op = PSY_CLOSURE_EMISSION;
    closure.roughness = PSY_INPUT_NONE;
    const float scalar = 2.0f, vector[3] = {0.25f, 0.5f, 0.75f};
    psy_material_desc material{};
    material.closures = &closure;
    material.closure_count = 1;
    material.scalars = &scalar;
    material.scalar_count = 1;
    material.vectors = vector;
    material.vector_count = 1;
    material.emission_sampling = 1u;
    psy_scene_desc desc{};
    desc.meshes = &mesh;
    desc.instances = &instance;
    desc.materials = &material;
    desc.mesh_count = desc.instance_count = desc.material_count = 1;
    psy_scene *scene = nullptr;
    CHECK(psy_scene_compile(context, &desc, &scene) == PSY_OK);
    CHECK(psy::host::ensure_light_tree(scene) == PSY_OK && scene->view.lt_node_count > 0u);

    auto view_lives = [&] {
        const psy::SceneView &v = scene->view;
        for (const void *p : {(const void *)v.scalars, (const void *)v.vectors, (const void *)v.baked,
                              (const void *)v.closures, (const void *)v.lt_nodes, (const void *)v.lt_emitters,
                              (const void *)v.lt_mapping, (const void *)v.lt_lookup})
            if (!fake::alive(p)) return false;
        return true;
    };
    auto holds = [&](float s, float v) {
        return scene->scalars[0] == s && scene->vectors[0] == v && scene->view.scalars[0] == s &&
               scene->view.vectors[0] == v;
    };
    const float next_scalar = 5.0f, next_vector[3] = {0.125f, 0.5f, 0.75f};
    const size_t held = fake::live.size();
    int rejected = 0;
    for (int k = 0;; ++k) {
        const psy::SceneView before = scene->view;
        fake::fail_in = k;
        const psy_status r =
            psy::host::rebind_parameters_versioned(scene, 0, &next_scalar, 1, next_vector, 1);
        if (r == PSY_OK) break;
        // the scene is as it was, also once the retired buffers are gone
        psy::host::release_retired(scene);
        CHECK(std::memcmp(&before, &scene->view, sizeof(before)) == 0);
        CHECK(view_lives() && holds(2.0f, 0.25f));
        CHECK(fake::live.size() == held);
        ++rejected;
    }
    fake::fail_in = -1;
    CHECK(rejected == 8);  // two parameter blocks, two baked tables, four of the light tree
    CHECK(view_lives() && holds(5.0f, 0.125f));
    psy::host::release_retired(scene);
    CHECK(view_lives() && fake::live.size() == held);
    psy_scene_destroy(scene);
    psy_context_destroy(context);
    CHECK(fake::live.empty());
    std::printf("ok\n");
    return 0;
}
