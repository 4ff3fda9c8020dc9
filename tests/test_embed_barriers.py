"""Layer 1's kernel between two tiles of a warp, read from its source (no GPU):
every lane reads all features of the warp's rows, so a barrier of the warp has
to stand between these reads and the next tile's writes on every path, whatever
the call's options are."""
import os
import re

from conftest import PKG


def _block(src, start):
    """The text between the braces that open at or after `start`."""
    a = src.index("{", start)
    depth = 0
    for i in range(a, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[a + 1:i]
    raise AssertionError("unbalanced braces")


def _top_level(text):
    """Statements outside nested braces, nested blocks as {}."""
    out, depth = [], 0
    for ch in text:
        depth -= ch == "}"
        if depth == 0:
            out.append(ch)
        depth += ch == "{"
    return "".join(out)


def test_a_warp_waits_between_reading_and_overwriting_its_features():
    with open(os.path.join(PKG, "csrc", "mlp.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    kernel = src.index("embed_kernel(EmbedArgs A)")
    loop = _block(src, src.index("for (int tile = ", kernel))
    assert loop.count("s_feat") == 2  # the writes' row and the sum
    write, read = loop.index("s_feat + "), loop.index("cols(s_feat[")
    assert write < read
    # what follows the loop over the tiles' sum, to the end of the pass
    rest = loop[read:]
    rest = rest[rest.index("}") + 1:]        # end of the loop over the rows
    rest = rest[rest.index("}") + 1:]        # end of the loop over the tiles
    before_branches = _top_level(rest).split("if (")[0]
    assert re.search(r"^\s*__sync(warp|threads)\(\);", before_branches), before_branches
