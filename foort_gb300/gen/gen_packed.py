"""Explicit-rounding forms of the generated right-hand sides, for packed FP32 arithmetic.

sm_103a has two-wide FP32 instructions (fma.rn.f32x2 and its siblings): one issue slot for
two fused multiply-adds. C++ operators on a pair type would not be contracted to fused
multiply-adds at all, while the compiler contracts the scalar bodies of
gen_christoffel.inc, so a pair body written with operators would round differently from
the scalar one. This script writes the bodies with every rounding spelled out (MUL, ADD,
FMA, RCP on a type T that is a float or a pair of floats), contracting as the compiler
does: a product joins a sum as an FMA where the sum is its only use, or where all of its
(fewer than five) uses are sums; with two such products the one that only this sum uses
joins, the left one first. A step's results are then the scalar body's bit for bit.

Products of the metric constants q[] alone are split off (FOORT_PACKED_CONST_*): a lane
computes them once per geodesic.

Usage: python gen_packed.py > ../csrc/gen_packed.inc   (reads ../csrc/gen_christoffel.inc)
"""
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = os.path.join(HERE, "..", "csrc", "gen_christoffel.inc")
TOKEN = re.compile(r"\s*(T\([0-9.e+-]+\)|q\[\d+\]|[A-Za-z_][\w.]*|[-+*()])")


class Graph:
    """Hash-consed expressions. A value is (sign, node): signs cost nothing."""

    def __init__(self):
        self.index, self.nodes, self.names, self.outputs = {}, [], {}, []

    def make(self, *key):
        if key not in self.index:
            self.index[key] = len(self.nodes)
            self.nodes.append(key)
        return self.index[key]

    def const(self, v):
        return (1 if v >= 0 else -1, self.make("const", abs(v)))

    def is_const(self, x):
        return self.nodes[x[1]][0] == "const"

    def mul(self, a, b):
        sign = a[0] * b[0]
        for x, y in ((a, b), (b, a)):
            if self.nodes[x[1]] == ("const", 1.0):
                return sign, y[1]
        key = ("mul", b[1], a[1])
        return sign, self.index[key] if key in self.index else self.make("mul", a[1], b[1])

    def add(self, a, b):
        key = ("add", b, a)
        return 1, self.index[key] if key in self.index else self.make("add", a, b)

    def operands(self, i):
        k = self.nodes[i]
        if k[0] == "mul":
            return [k[1], k[2]]
        if k[0] == "add":
            return [k[1][1], k[2][1]]
        return [k[1][1]] if k[0] == "rcp" else []

    def parse(self, text):
        toks, at = TOKEN.findall(text), [0]

        def peek():
            return toks[at[0]] if at[0] < len(toks) else None

        def take():
            at[0] += 1
            return toks[at[0] - 1]

        def total():
            x = product()
            while peek() in ("+", "-"):
                sign = 1 if take() == "+" else -1
                y = product()
                x = self.add(x, (sign * y[0], y[1]))
            return x

        def product():
            x = factor()
            while peek() == "*":
                take()
                x = self.mul(x, factor())
            return x

        def factor():
            t = take()
            if t == "-":
                x = factor()
                return -x[0], x[1]
            if t in ("(", "rcp"):
                if t == "rcp":
                    take()
                x = total()
                assert take() == ")", text
                return (1, self.make("rcp", x)) if t == "rcp" else x
            if t.startswith("T("):
                return self.const(float(t[2:-1]))
            return self.names.get(t) or (1, self.make("leaf", t))

        x = total()
        assert at[0] == len(toks), text
        return x


def read_body(name):
    g = Graph()
    text = re.search(r"#define FOORT_MIXED_BODY_%s \\\n((?:.*\\\n)*.*\n)" % name, open(SOURCE).read()).group(1)
    for line in text.strip().split("\n"):
        line = line.rstrip("\\").strip().rstrip(";")
        m = re.match(r"const T (\w+) = (.*)$", line)
        if m:
            g.names[m.group(1)] = g.parse(m.group(2))
            continue
        target, expr = line.split(" = ", 1)
        if target != "grr":
            g.outputs.append((target, g.parse(expr)))
    return g


def reachable(g):
    seen, todo = set(), [x[1] for _, x in g.outputs]
    while todo:
        i = todo.pop()
        if i not in seen:
            seen.add(i)
            todo += g.operands(i)
    return seen


def contraction(g):
    """add node -> index (0 or 1) of the product operand that joins it, or None."""
    live, users = reachable(g), {}

    def positive(x):
        return x[0] > 0 or g.is_const(x)

    for i in live:
        k = g.nodes[i]
        kind = "add" if k[0] == "add" and positive(k[1]) and positive(k[2]) else "other"
        for o in g.operands(i):
            users.setdefault(o, []).append(kind)
    for _, x in g.outputs:
        users.setdefault(x[1], []).append("other")
    out = {}
    for i in live:
        k = g.nodes[i]
        if k[0] != "add":
            continue
        ops = [x[1] for x in k[1:]]
        product = [g.nodes[o][0] == "mul" for o in ops]
        single = [p and len(users[o]) == 1 for p, o in zip(product, ops)]
        sums = [p and len(users[o]) < 5 and all(u == "add" for u in users[o]) and positive(k[1]) and positive(k[2])
                for p, o in zip(product, ops)]
        out[i] = 0 if single[0] else 1 if single[1] else 0 if sums[0] else 1 if sums[1] else None
    return out


def emit(name):
    g = read_body(name)
    fuse, live = contraction(g), reachable(g)
    only_q = {}

    def constant(i):
        """Made of q[] alone."""
        if i not in only_q:
            k = g.nodes[i]
            only_q[i] = k[1].startswith("q[") if k[0] == "leaf" else k[0] == "mul" and all(map(constant, k[1:]))
        return only_q[i]

    needed = sorted({o for i in live if not constant(i) for o in operands_after(g, fuse, i) if constant(o)})
    consts, body, done = [], [], {}

    def value(i, lines):
        if i in done:
            return done[i]
        k = g.nodes[i]
        if k[0] == "leaf":
            return k[1]
        if k[0] == "const":
            return "K(%sf)" % k[1]
        if k[0] == "mul":
            text = "MUL(%s, %s)" % (value(k[1], lines), value(k[2], lines))
        elif k[0] == "rcp":
            text = "RCP(%s)" % signed(k[1], lines)
        elif fuse[i] is None:
            text = "ADD(%s, %s)" % (signed(k[1], lines), signed(k[2], lines))
        else:
            m, o = (k[1], k[2]) if fuse[i] == 0 else (k[2], k[1])
            a, b = g.nodes[m[1]][1:]
            text = "FMA(%s%s, %s, %s)" % ("-" if m[0] < 0 else "", value(a, lines), value(b, lines), signed(o, lines))
        lines.append("const T n%d = %s;" % (i, text))
        done[i] = "n%d" % i
        return done[i]

    def signed(x, lines):
        return ("-" if x[0] < 0 else "") + value(x[1], lines)

    for slot, i in enumerate(needed):
        text = value(i, consts)
        consts.append("k[%d] = %s;" % (slot, text))
    consts = [line.replace("const T ", "const float ") for line in consts]
    for slot, i in enumerate(needed):
        done[i] = "B(%d)" % slot
    body += ["%s = %s;" % (target, signed(x, body)) for target, x in g.outputs]
    print("// %d operations on T" % sum(line.startswith("const") for line in body))
    print("#define FOORT_PACKED_SLOTS_%s %d" % (name, len(needed)))
    print("#define FOORT_PACKED_CONST_%s \\" % name)
    print(" \\\n".join("    " + line for line in consts or [";"]))
    print("#define FOORT_PACKED_BODY_%s \\" % name)
    print(" \\\n".join("    " + line for line in body))
    print()


def operands_after(g, fuse, i):
    """Operands of node i once products have joined sums."""
    k = g.nodes[i]
    if k[0] == "add" and fuse[i] is not None:
        m, o = (k[1], k[2]) if fuse[i] == 0 else (k[2], k[1])
        return list(g.nodes[m[1]][1:]) + [o[1]]
    return g.operands(i)


def main():
    print("// Explicit-rounding bodies of the inlined plugins.")
    print("// Generated by foort_gb300/gen/gen_packed.py -- do not edit.")
    print("// In: r, dp = r - r_+, dm = r - r_-, s = sin(theta), c = cos(theta) of type T, B(i): the")
    print("// lane's constant i as a T. Out: dr, dh, gu as in gen_christoffel.inc.")
    for name in ("KERR", "FLAT"):
        emit(name)


if __name__ == "__main__":
    main()
