"""Every copy, fill and launch of the library goes through a stream that it names.  A context's stream is
created non-blocking, so nothing orders it with the legacy stream, and a copy from pageable memory
on that one may still be under way when the call returns: a kernel launched on the context's stream
right after it can read what was in the memory before."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "galfast_b200", "csrc")


def sources():
    for fn in sorted(glob.glob(os.path.join(CSRC, "*"))):
        if fn.endswith((".cu", ".cuh", ".h", ".cpp")):
            with open(fn) as f:
                yield os.path.basename(fn), re.sub(r"/\*.*?\*/|//[^\n]*", "", f.read(), flags=re.S)


def test_no_copy_or_fill_on_the_legacy_stream():
    found = [(name, m.group(0)) for name, text in sources() for m in re.finditer(r"\bcuda(Memcpy|Memset)(2D|3D|ToSymbol|FromSymbol)?\s*\(", text)]
    assert not found


def test_every_launch_names_its_stream():
    launches = [(name, m.group(1)) for name, text in sources() for m in re.finditer(r"<<<(.*?)>>>", text, flags=re.S)]
    assert len(launches) > 30
    for name, args in launches:
        assert re.search(r",\s*(s|st|ctx->stream|s->ctx->stream)\s*$", args), (name, args)
