"""A renderer's side streams are made by the calls that launch waves on them, each
of those calls, and not with the renderer: read from the source, since no
result depends on it."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "photon_gb300", "csrc", "renderer.cpp")


def _body(text, head):
    start = text.index("{", text.index(head))
    depth, end = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
            return text[start:end]


def test_side_streams_belong_to_the_waves():
    text = open(SRC).read()
    create = _body(text, "int phc_create(phc_renderer **out)")
    assert "side[" not in create and "ensure_sides" not in create
    for head, recorded in (("void render_impl(", r"\brecord_wave\("), ("void render_batch_impl(", r"\brecord_batch_wave\("),
                           ("void adjoint_impl(", r"\brecord_wave\(")):
        body = _body(text, head)
        made = body.index("ensure_sides(")
        assert made < re.search(recorded, body).start(), head
        if "cudaStreamBeginCapture" in body:
            assert made < body.index("cudaStreamBeginCapture"), head
