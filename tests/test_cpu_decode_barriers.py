"""The hardware barriers of the decode kernel, read from its source: none is used with two numbers of threads. In normal operation the
exchanges between two uses hide such a clash; once a wait has given up they are skipped, and a clash could then block the kernel for good."""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "gradients.c_b200", "csrc", "decode_cluster.cu")


def barrier_threads(text):
    """{barrier: {numbers of threads it is used with}} over all units u (up to eight halves apart) and sums ou (two)."""
    names = {}
    for decl in re.findall(r"constexpr (?:int|uint32_t) ((?:DC_\w+ = [^;]+));", text):
        for name, value in re.findall(r"(DC_\w+) = ([^,;]+)", decl):
            try:
                names[name] = int(eval(re.sub(r"(\d)U\b", r"\1", value), {}, names))
            except (SyntaxError, NameError):
                pass
    uses = {0: {(names["DC_WARPS"] + names["DC_PRODUCERS"]) * 32}}
    found = re.findall(r'"bar\.(?:sync|arrive) (\w+|%0), (\d+|%\d);" ::([^;]*?): "memory"', text)
    assert len(found) >= 4
    for barrier, count, operands in found:
        values = [re.sub(r"\(uint32_t\)|(?<=\d)U\b", "", v) for v in re.findall(r'"[rn]"\(((?:[^()]|\([^()]*\))*)\)', operands)]
        if barrier != "%0":
            values.insert(0, barrier)
        for u in range(8):
            for ou in range(2):
                at = int(eval(values[0], {}, dict(names, u=u, ou=ou)))
                threads = int(count) if count.isdigit() else int(eval(values[1], {}, dict(names)))
                uses.setdefault(at, set()).add(threads)
    return uses


def test_no_barrier_has_two_numbers_of_threads():
    uses = barrier_threads(open(SRC).read())
    assert max(uses) < 16 and {t for s in uses.values() for t in s} >= {64, 256, 512}
    assert all(len(s) == 1 for s in uses.values()), uses
