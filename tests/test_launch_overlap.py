"""Kernels that are set up while the kernel before them still runs.

Launched with programmatic stream serialization, a kernel may start before its
predecessor has finished; it waits for it in its first statement (pdl_begin).
A __restrict__ pointer tells the compiler that nobody writes what it points
to as long as the kernel runs, so loads through it may be moved above that
wait.  Hence

 * no kernel declares a __restrict__ pointer of its own in its body (what it
   points to may be the predecessor's output), and neither does the transfer
   kernel in its parameters;
 * the job descriptors are a __restrict__ parameter only of kernels that cannot
   start before the descriptors' upload has finished: not of those that may
   follow the upload directly.  (The kernel after such a one starts only when
   that one has passed its own wait.)

A check of the sources: what the compiler makes of it differs by version."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "luda_b200", "csrc")

# the launches that may be the first after the descriptors' upload, with their
# first kernel
AFTER_UPLOAD = {
    "launch_table_index_count": "k_table_index_count",  # parse
    "launch_parse_done": "k_parse_done",                # parse of a batch without tables
    "launch_block_decode": "k_decode_walk",             # after the parse
    "launch_entries_from_offsets": "k_entries_from_offsets",  # flush encoder
}


def _sources():
    out = {}
    for p in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(p) as f:
            out[os.path.basename(p)] = re.sub(r"//[^\n]*", "", f.read())
    return out


def _body(text, at):
    """The braces' content from the first brace at or after `at`."""
    i = text.index("{", at)
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == "{") - (text[j] == "}")
        if not depth:
            return text[i:j]
    raise AssertionError("unbalanced braces")


def _kernels():
    """name -> (parameters, body) of every kernel that begins with the wait."""
    found = {}
    for text in _sources().values():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(([^)]*)\)\s*\{", text):
            body = _body(text, m.end() - 1)
            if "pdl_begin()" in body:
                found[m.group(1)] = (m.group(2), body)
    return found


def test_every_overlapping_kernel_is_found():
    k = _kernels()
    assert len(k) > 30 and set(AFTER_UPLOAD.values()) <= set(k) and "k_xfer" in k


def test_no_restrict_in_bodies():
    assert [n for n, (_, body) in _kernels().items() if "__restrict__" in body] == []


def test_no_restrict_right_after_a_writer():
    k = _kernels()
    first = set(AFTER_UPLOAD.values()) | {"k_xfer"}
    assert [n for n in sorted(first) if "__restrict__" in k[n][0]] == []


def test_first_kernels_are_the_listed_ones():
    text = "\n".join(_sources().values())
    for fn, kernel in AFTER_UPLOAD.items():
        body = _body(text, text.index(f"void {fn}(const Batch& bt, cudaStream_t st) {{"))
        assert re.search(r"launch(?:_clusters)?\(\s*(\w+)", body).group(1) == kernel, fn
    # the engine's launches after an upload, up to the next wait of the host
    eng = _sources()["lc_engine.cu"]
    tail = _body(eng, eng.index("void launch_tail("))
    assert re.findall(r"launch_\w+", tail)[0] == "launch_block_decode"
    build = _body(eng, eng.index("void run_build("))
    after = build[build.rindex("slot.to_device("):]
    assert re.findall(r"launch_\w+", after)[0] == "launch_entries_from_offsets"
    batch = _body(eng, eng.index("void run_batch("))
    up = [m.end() for m in re.finditer(r"slot\.to_device\(", batch)]
    calls = {re.search(r"(launch_\w+|run_tail)\(", batch[a:]).group(1) for a in up}
    assert calls == {"launch_table_index_count", "run_tail"}, calls
