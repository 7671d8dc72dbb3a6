"""A process loads a translation unit's device image when it first launches a kernel of it, all
variants of all its kernels at once.  Most of the library's device code are the variants of the walk
and the pair kernels: the two math modes are instantiated in different translation units, and the
walk's tile shapes other than the default in a third."""
import os
import re

from akuaengine_gb300 import build

KERNELS = "search|density_lambda|delta_correct|delta_final|vorticity|confine|xsph"


def test_math_modes_and_tile_shapes_have_images_of_their_own():
    modes, shapes = {}, set()
    for path in build.sources():
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        found = set(re.findall(r"\benqueue_pairs<\s*(\w+)", text))
        found |= set(re.findall(r"\bk_(?:%s)<\s*(\w+)" % KERNELS, text))
        if found:
            modes[os.path.basename(path)] = found
        if "launch_search_shape<" in text:
            shapes.add(os.path.basename(path))
    assert sorted(modes.values(), key=sorted) == [{"false"}, {"true"}], modes
    assert len(shapes) == 1 and not shapes & set(modes), shapes
