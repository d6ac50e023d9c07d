"""The warp-wide Tensor Memory instructions bring their warp together first.

Every lane of a warp has to execute a ``.sync.aligned`` instruction together,
and the wrappers are called behind branches that depend on the lane (a column
past a ragged edge, a row past the field, a strided loop's last round).  Nothing
at run time shows a warp that was still split, so the sources are read: each
function with such an instruction calls ``__syncwarp()`` before the first one."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xlumina_gb300", "csrc")
ALIGNED = re.compile(r'"tcgen05\.[^"]*\.sync\.aligned')


def _functions(text):
    """(name, body) of every function at file scope: from a line that starts
    with ``__device__`` or ``template`` to the closing brace in column 0, or a
    function on one line."""
    for m in re.finditer(r"^(?:template[^\n]*\n?)?[^\n]*__device__[^\n;]*?(\w+)\(.*?(?:^\}|\}$)", text, re.M | re.S):
        yield m.group(1), m.group(0)


def test_every_aligned_instruction_follows_a_syncwarp():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = open(path).read()
        inside = 0
        for name, body in _functions(text):
            hits = ALIGNED.findall(body)
            if hits:
                inside += len(hits)
                sync = body.find("__syncwarp();")
                assert 0 <= sync < ALIGNED.search(body).start(), f"{os.path.basename(path)}: {name}"
        assert inside == len(ALIGNED.findall(text)), f"{os.path.basename(path)}: outside the functions that were read"
        seen += inside
    assert seen >= 6
