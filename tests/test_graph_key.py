"""Every buffer that a learned frame sizes belongs to the key of its recorded graph (a reallocated one must not replay)."""
import os
import re

from conftest import PKG


def _body(text, head):
    a = text.index(head)
    return text[a:text.index("\n}\n", a)]


def test_recorded_frame_key_names_every_buffer_the_frame_sizes():
    with open(os.path.join(PKG, "csrc", "pf_api.cu")) as f:
        text = f.read()
    sized = set()
    for head in ("int begin_frame(", "int stage_setup(", "int bin_and_composite(", "int render_learned_frame("):
        sized |= set(re.findall(r"c->(\w+)\.ensure\(", _body(text, head)))
    key = _body(text, "std::vector<void *> frame_buffers(")
    assert len(sized) > 20
    assert sized <= set(re.findall(r"&c->(\w+)", key))
