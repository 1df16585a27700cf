"""A batch's kernels run on a stream that does not wait for the legacy default
stream, and the synchronous forms of copies and fills work on the latter: a
copy from pageable memory returns once its source has been staged, a fill of
device memory at once.  So whatever writes device memory in the library does
so on the batch's (or the caller's) stream; the synchronous forms only read
results back, behind a wait for the stream."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vlasiator_b200", "csrc")


def _calls(name):
    """Every call of the function `name` in the sources: (file, line, arguments as text)."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"\b%s\s*\(" % name, text):
            depth, at = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            yield os.path.basename(path), text.count("\n", 0, m.start()) + 1, text[m.end():at - 1]


def test_no_write_on_the_legacy_stream():
    writes = [c for c in _calls("cudaMemset")]
    writes += [c for c in _calls("cudaMemcpy") if "cudaMemcpyDeviceToHost" not in c[2]]
    assert not writes, writes


def test_async_calls_name_a_stream():
    """The asynchronous forms take the legacy stream too where their last argument is left out or zero."""
    for name, n_args in (("cudaMemsetAsync", 4), ("cudaMemcpyAsync", 5)):
        found = 0
        for where in _calls(name):
            depth, args = 0, [""]
            for ch in where[2]:
                depth += {"(": 1, "[": 1, "{": 1, ")": -1, "]": -1, "}": -1}.get(ch, 0)
                if ch == "," and depth == 0:
                    args.append("")
                else:
                    args[-1] += ch
            assert len(args) == n_args and re.search(r"\b(s|stream)$", args[-1].strip()), where
            found += 1
        assert found
