"""Every entry point of the device library says whether a recorded run may repeat it."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# nothing of theirs would be missing from a repeated run
UNMARKED = {
    "wdc_create", "wdc_destroy",                              # a context's beginning and end
    "wdc_last_error", "wdc_stats", "wdc_reset_stats",         # read and reset counters of the host
    "wdc_range_push", "wdc_range_pop",                        # ranges of a profiler; such runs are not recorded
    "wdc_tape_begin", "wdc_tape_end", "wdc_tape_destroy",     # the recording itself
}
BY = {"wdc_upload_async": "upload_async", "wdc_upload_fresh_async": "upload_async"}   # marked in what they call


def _body(source, start):
    depth, i = 1, start
    while depth:
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        i += 1
    return source[start:i]


def test_entry_points_are_marked():
    seen, unmarked = set(), set()
    for path in glob.glob(os.path.join(ROOT, "webdnn_b200", "csrc", "*.cu")):
        source = open(path).read()
        for m in re.finditer(r'extern "C" [\w \*]+?\b(wdc_\w+)\(([^)]*)\)\s*\{', source):
            if "wdc_context*" not in m.group(2):
                continue
            seen.add(m.group(1))
            body = _body(source, m.end())
            if m.group(1) in BY:
                f = re.search(r"static int %s\([^)]*\)\s*\{" % BY[m.group(1)], source)
                assert BY[m.group(1)] + "(" in body
                body = _body(source, f.end())
            if not re.search(r"WDC_TAPE\(|WDC_NO_TAPE\(|TapeScope ", body):
                unmarked.add(m.group(1))
    header = open(os.path.join(ROOT, "include", "webdnn_cuda.h")).read()
    declared = {m.group(1) for m in re.finditer(r"\b(wdc_\w+)\(([^;]*?)\);", header) if "wdc_context*" in m.group(2)}
    assert declared <= seen, declared - seen
    assert unmarked == UNMARKED


def test_taped_calls_repeat_themselves():
    """WDC_TAPE names the function that it stands in."""
    for path in glob.glob(os.path.join(ROOT, "webdnn_b200", "csrc", "*.cu")):
        source = open(path).read()
        for m in re.finditer(r'extern "C" int (wdc_\w+)\([^)]*\)\s*\{', source):
            for named in re.findall(r"WDC_TAPE\(ctx, (\w+)", _body(source, m.end())):
                assert named == m.group(1)
