// What the host makes of a scene before any device work, for test_plain_class.py.
#include "../repackshot_b200/csrc/rtg_scene.h"

#include <string>

using namespace rtg;

// SceneDev::plain of an RSB scene; 2 when it does not load.
extern "C" uint32_t host_plain(const uint8_t* bytes, uint64_t len) {
    HScene scene;
    Flat flat;
    std::string error;
    if (!parse_rsb(bytes, len, scene, error) || !flatten_scene(scene, flat, error)) return 2;
    return flat.scene.plain;
}
