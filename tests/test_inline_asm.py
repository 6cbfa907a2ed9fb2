"""Inline assembly in fp4_post_b200/csrc against the contract that the compiler holds it to: a statement that reads or writes memory is
volatile (else it may move in front of the wait for the kernel that wrote that memory, or of a barrier), and an output that is written
before the last input is read is marked (else it may get that input's register)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "fp4_post_b200" / "csrc"
STATEMENT = re.compile(r"\basm\s*(volatile)?\s*\(")
TEXT = re.compile(r'"((?:[^"\\]|\\.)*)"')
MEMORY = re.compile(r"(^|[\s;{])(ld|st|red|atom|cp|mbarrier|tcgen05|multimem|prefetch|fence|membar|griddepcontrol)\b[.\w:]*")


def body(source, start):
    """What stands between the parentheses of the statement whose opening one ends at `start`."""
    depth, i, quoted = 1, start, False
    while depth:
        c = source[i]
        if quoted and c == "\\":
            i += 1
        elif c == '"':
            quoted = not quoted
        elif not quoted:
            depth += (c == "(") - (c == ")")
        i += 1
    return source[start:i - 1]


def statements():
    for path in sorted(CSRC.glob("*.cu*")):
        source = path.read_text()
        for m in STATEMENT.finditer(source):
            line = source[:m.start()].count("\n") + 1
            yield f"{path.name}:{line}", bool(m.group(1)), body(source, m.end())


def parts(text):
    """Template, constraints of the outputs and of the inputs."""
    fields, depth, quoted, at = [""], 0, False, 0
    while at < len(text):
        c = text[at]
        if c == '"':
            quoted = not quoted
        if not quoted:
            depth += (c == "(") - (c == ")")
            if c == ":" and depth == 0:
                fields += [""] * (2 if text[at:at + 2] == "::" else 1)
                at += 2 if text[at:at + 2] == "::" else 1
                continue
        fields[-1] += c
        at += 1
    template = "".join(TEXT.findall(fields[0])).replace("\\n", "\n").replace("\\t", " ")
    constraints = [re.findall(r'"([^"]*)"\s*\(', f) for f in fields[1:3]] + [[], []]
    return template, constraints[0], constraints[1]


def test_memory_is_touched_by_volatile_statements_only():
    seen = 0
    for where, volatile, text in statements():
        template = parts(text)[0]
        touches = MEMORY.search(template) is not None
        seen += touches
        assert volatile or not touches, f"{where}: {template!r}"
    assert seen > 30


def test_outputs_written_before_the_last_input_is_read_are_marked():
    seen = 0
    for where, _, text in statements():
        template, outputs, inputs = parts(text)
        steps = [s for s in template.replace("%%", "").split(";") if re.search(r"%\d", s)]
        if len(steps) < 2:
            continue
        seen += 1
        last_read = max((i for i, s in enumerate(steps) for n in re.findall(r"%(\d+)", s) if int(n) >= len(outputs)), default=-1)
        for n, constraint in enumerate(outputs):
            first_write = min((i for i, s in enumerate(steps) if re.search(rf"%{n}\b", s)), default=len(steps))
            assert "&" in constraint or "+" in constraint or first_write >= last_read, f"{where}: output {n} of {template!r}"
    assert seen >= 5
