"""Explicit-rounding forms of the generated right-hand sides, for packed FP32 arithmetic.

sm_103a has two-wide FP32 instructions (fma.rn.f32x2 and its siblings): one issue slot for
two fused multiply-adds. C++ operators on a pair type would not be contracted to fused
multiply-adds at all, while the compiler contracts the scalar bodies of
gen_christoffel.inc, so a pair body written with operators would round differently from
the scalar one. This script writes the bodies with every rounding spelled out (MUL, ADD,
FMA, RCP on a type T that is a float or a pair of floats), contracting as the compiler
does: a product joins a sum as an FMA where all of its (fewer than five) uses are sums, or
where the sum comes far behind it; of two such products the left one. A step's results are then the scalar body's bit for bit.

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


# Where the compiled Johannsen body departs from contraction()'s rule, found by comparing
# 262,144 evaluations (four spins and alpha13, r_+ + 0.002 to 1000) bit for bit: sum -> the
# operand whose product joins it.
EXCEPTIONS = {"JOHANNSEN": {89: 1, 614: 1, 1036: 1, 1045: 1}}
FAR = 500  # operations between a product and a sum that make the compiler fuse it all the same


def contraction(g, name):
    """add node -> index (0 or 1) of the product operand that joins it, or None. Sums are
    taken from the last to the first: a sum that has taken a product no longer counts as a
    sum for its other operand."""
    live, users, order = reachable(g), {}, {}

    def positive(x):
        return x[0] > 0 or g.is_const(x)

    at = 0
    for i in sorted(live):
        k = g.nodes[i]
        if k[0] in ("mul", "add", "rcp"):
            order[i] = at
            at += 4 if k[0] == "rcp" else 1
        kind = "add" if k[0] == "add" and positive(k[1]) and positive(k[2]) else "other"
        for o in g.operands(i):
            users.setdefault(o, []).append([i, kind])
    for _, x in g.outputs:
        users.setdefault(x[1], []).append([None, "other"])

    def joins(m, total):
        if g.nodes[m][0] != "mul" or len(users[m]) >= 5:
            return False
        if all(kind == "add" for _, kind in users[m]):
            return True
        if order[total] - order[m] < FAR:
            return False
        return any(g.nodes[o][0] == "const" or any(u is None or order[u] > order[total] for u, _ in users[o])
                   for o in g.nodes[m][1:])

    out = {}
    for i in sorted((i for i in live if g.nodes[i][0] == "add"), reverse=True):
        k = g.nodes[i]
        ops = [x[1] for x in k[1:]]
        if positive(k[1]) and positive(k[2]):
            join = next((n for n in (0, 1) if joins(ops[n], i)), None)
        else:  # a difference takes a product that only it uses
            join = next((n for n in (0, 1) if g.nodes[ops[n]][0] == "mul" and len(users[ops[n]]) == 1), None)
        join = EXCEPTIONS.get(name, {}).get(i, join)
        out[i] = join
        if join is not None:
            users[ops[join]] = [u for u in users[ops[join]] if u[0] != i]
            for o in g.nodes[ops[join]][1:]:
                users[o].append([i, "fma"])
            for u in users[ops[1 - join]]:
                if u[0] == i:
                    u[1] = "fma"
    return out


class Ops:
    """The operations of a contracted body, each once. Values are ("c", number) or
    ("v", sign, text); operations with a zero or a one fold away, exactly."""

    def __init__(self, g, fuse, zeros):
        self.g, self.fuse, self.zeros = g, fuse, zeros
        self.done, self.index, self.list = {}, {}, []

    def op(self, *key):
        if key not in self.index:
            self.index[key] = "n%d" % len(self.list)
            self.list.append((self.index[key], key))
        return self.index[key]

    @staticmethod
    def text(v):
        if v[0] == "c":
            return ("-" if v[1] < 0 else "") + "K(%rf)" % abs(v[1])
        return ("-" if v[1] < 0 else "") + v[2]

    @staticmethod
    def negated(v):
        return ("c", -v[1]) if v[0] == "c" else ("v", -v[1], v[2])

    def factors(self, a, b):
        """(sign, a, b) with the signs taken out, or the product where it folds."""
        if ("c", 0.0) in (a, b):
            return ("c", 0.0)
        for x, y in ((a, b), (b, a)):
            if x[0] == "c" and abs(x[1]) == 1.0:
                return y if x[1] > 0 else self.negated(y)
        sign, texts = 1, []
        for v in (a, b):
            texts.append(self.text(v).lstrip("-"))
            sign *= -1 if self.text(v).startswith("-") else 1
        return sign, texts[0], texts[1]

    def mul(self, a, b):
        f = self.factors(a, b)
        if f[0] in ("c", "v"):
            return f
        sign, x, y = f
        return "v", sign, self.index.get(("MUL", y, x)) or self.op("MUL", x, y)

    def add(self, a, b):
        if a == ("c", 0.0):
            return b
        return a if b == ("c", 0.0) else ("v", 1, self.op("ADD", self.text(a), self.text(b)))

    def fma(self, a, b, c):
        if c == ("c", 0.0):
            return self.mul(a, b)
        f = self.factors(a, b)
        if f[0] in ("c", "v"):
            return self.add(f, c)
        return "v", 1, self.op("FMA", ("-" if f[0] < 0 else "") + f[1], f[2], self.text(c))

    def signed(self, x):
        v = self.value(x[1])
        return v if x[0] > 0 else self.negated(v)

    def value(self, i):
        if i in self.done:
            return self.done[i]
        k = self.g.nodes[i]
        if k[0] == "leaf":
            v = ("c", 0.0) if k[1] in self.zeros else ("v", 1, k[1])
        elif k[0] == "const":
            v = ("c", k[1])
        elif k[0] == "mul":
            v = self.mul(self.value(k[1]), self.value(k[2]))
        elif k[0] == "rcp":
            x = self.signed(k[1])
            v = ("c", 1.0) if x == ("c", 1.0) else ("v", 1, self.op("RCP", self.text(x)))
        elif self.fuse[i] is None:
            v = self.add(self.signed(k[1]), self.signed(k[2]))
        else:
            m, o = (k[1], k[2]) if self.fuse[i] == 0 else (k[2], k[1])
            x, y = (self.value(j) for j in self.g.nodes[m[1]][1:])
            v = self.fma(x if m[0] > 0 else self.negated(x), y, self.signed(o))
        self.done[i] = v
        return v


def emit(name, label=None, zeros=()):
    g = read_body(name)
    ops = Ops(g, contraction(g, name), zeros)
    outputs = [(target, ops.text(ops.signed(x))) for target, x in g.outputs]
    made = dict(ops.list)
    word = re.compile(r"\bn\d+\b|q\[\d+\]")

    def inputs(key):
        return [w for arg in key[1:] for w in word.findall(arg)]

    live, todo = set(), [w for _, e in outputs for w in word.findall(e)]
    while todo:
        w = todo.pop()
        if w not in live:
            live.add(w)
            todo += inputs(made[w]) if w in made else []
    # the lane's constants: made of q[] alone and used by the rest, but for small multiples
    only_q = {w for w in live if w.startswith("q[")}
    for w, key in ops.list:
        if w in live and not re.search(r"\b(r|dp|dm|s|c)\b", " ".join(key[1:])) and key[0] != "RCP" \
                and all(v in only_q for v in inputs(key)):
            only_q.add(w)
    multiple = {w for w in only_q if w in made and made[w][0] == "MUL" and made[w][1].startswith("K(")}
    kept, seen = [], set()

    def need(w):
        if w not in only_q or w in seen:
            return
        seen.add(w)
        if w in multiple:
            for v in inputs(made[w]):
                need(v)
        else:
            kept.append(w)

    rest = [w for w, _ in ops.list if w in live and w not in only_q]
    for w in rest:
        for v in inputs(made[w]):
            need(v)
    order = {w: n for n, (w, _) in enumerate(ops.list)}
    kept.sort(key=lambda w: order.get(w, -1))
    slot = {w: "B(%d)" % n for n, w in enumerate(kept)}
    consts, have = [], set()

    def const_line(w):
        if w in made and w not in have:
            have.add(w)
            for v in inputs(made[w]):
                const_line(v)
            consts.append("const float %s = %s(%s);" % (w, made[w][0], ", ".join(made[w][1:])))

    for n, w in enumerate(kept):
        const_line(w)
        consts.append("k[%d] = %s;" % (n, w))

    def put(text):
        return word.sub(lambda m: slot.get(m.group(0), m.group(0)), text)

    body = ["const T %s = %s(%s);" % (w, key[0], ", ".join(map(put, key[1:]))) for w, key in ops.list
            if w in live and (w not in only_q or w in multiple and w in seen)]
    print("// %d operations on T" % len(body))
    label = label or name
    print("#define FOORT_PACKED_SLOTS_%s %d" % (label, len(kept)))
    print("#define FOORT_PACKED_CONST_%s \\" % label)
    print(" \\\n".join("    " + line for line in consts or [";"]))
    print("#define FOORT_PACKED_BODY_%s \\" % label)
    print(" \\\n".join("    " + line for line in body + ["%s = %s;" % (t, put(e)) for t, e in outputs]))
    print()


def main():
    print("// Explicit-rounding bodies of the inlined plugins.")
    print("// Generated by foort_gb300/gen/gen_packed.py -- do not edit.")
    print("// In: r, dp = r - r_+, dm = r - r_-, s = sin(theta), c = cos(theta) of type T, B(i): the")
    print("// lane's constant i as a T. Out: dr, dh, gu as in gen_christoffel.inc.")
    for name in ("KERR", "FLAT"):
        emit(name)
    # Johannsen's metric with alpha13 alone: the shipped configurations and the studies of
    # one deviation at a time
    emit("JOHANNSEN", "JOHANNSEN13", ("q[2]", "q[3]", "q[4]"))


if __name__ == "__main__":
    main()
