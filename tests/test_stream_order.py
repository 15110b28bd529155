"""Device memory is cleared on the stream that uses it next.

The context's streams do not wait for the default stream, and a cudaMemset on
device memory returns before it has run: a buffer cleared that way could be
cleared while, or after, a kernel has used it, or under the next owner of a
reused block.  That cannot be run for (it would corrupt the kernels' own
counters), so the sources are read instead."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turbo-cat_b200", "csrc")


def _code(path):
    text = re.sub(r"/\*.*?\*/", " ", open(path).read(), flags=re.S)
    return re.sub(r"//[^\n]*", " ", text)


def test_no_clearing_on_the_default_stream():
    files = sorted(glob.glob(os.path.join(CSRC, "*")))
    assert files
    for path in files:
        code = _code(path)
        assert not re.search(r"\bcudaMemset(2D|3D)?\s*\(", code), path
        # every asynchronous clear names a stream (four arguments)
        for m in re.finditer(r"\bcudaMemsetAsync\s*\(", code):
            depth, args, i = 1, 1, m.end()
            while depth:
                ch = code[i]
                depth += ch in "([{"
                depth -= ch in ")]}"
                args += ch == "," and depth == 1
                i += 1
            assert args == 4, (path, code[m.start():i])
