"""Kernels launched by launch_chained may start before the work ahead of them in the
stream has ended.  Completion is transitive along the stream only if each of them
waits (grid_wait) in all its threads: no thread may return before the wait."""

import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "spectral-kernel-benchmarks_b200", "csrc", "*.cu")))


def _block(text, start):
    """Text of the brace block that opens at or after `start`."""
    begin = text.index("{", start)
    depth = 0
    for i in range(begin, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[begin:i + 1]
    raise ValueError("unbalanced braces")


def _without_lambdas(body):
    lambda_head = re.compile(r"\[[&=]?\]\s*(\((?:[^()]|\([^()]*\))*\))?\s*(->\s*[\w*]+\s*)?(?=\{)")
    while (m := lambda_head.search(body)) is not None:
        inner = _block(body, m.end())
        body = body[:m.start()] + body[m.end() + len(inner):]
    return body


def _chained_kernels():
    found = {}
    for path in SOURCES:
        text = re.sub(r"//[^\n]*", "", open(path).read())
        names = set()
        for call in re.finditer(r"launch_chained\(\s*(\w+)", text):
            if call.group(1) == "kernel":
                assigned = list(re.finditer(r"auto kernel = ([^;]+);", text[:call.start()]))[-1].group(1)
                names |= set(re.findall(r"\w+_kernel", assigned))
            else:
                names.add(call.group(1))
        for name in names:
            head = re.search(r"\b%s\s*\(" % name, text)
            assert head and "__global__" in text[max(0, head.start() - 300):head.start()], name
            found[os.path.basename(path), name] = _without_lambdas(_block(text, text.index(")", head.end())))
    return found


def test_every_chained_kernel_waits_in_all_its_threads():
    kernels = _chained_kernels()
    assert len(kernels) >= 12
    for (path, name), body in kernels.items():
        assert "grid_wait();" in body, (path, name)
        before = body[:body.index("grid_wait();")]
        assert not re.search(r"\breturn\b", before), (path, name)
