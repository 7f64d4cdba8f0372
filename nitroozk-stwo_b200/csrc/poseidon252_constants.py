"""Writes poseidon252_constants.inc and poseidon252_constants_host.inc: the
constants of Starknet's Poseidon (the Hades permutation of starknet-crypto
0.6.2, which the reference's Poseidon252 Merkle hasher and channel call),
Montgomery form with R = 2^256: 8 little-endian 32-bit limbs per field
element in the device layout of poseidon252.cu, 4 little-endian 64-bit limbs
for the prover's host channel (prover/felt252_host.h).

Field: p = 2^251 + 17·2^192 + 1. Round constants, the published rule:
SHA-256 of "Hades" followed by the decimal index, as a big-endian integer,
reduced mod p, for index 3·round + element, 91 rounds. The partial rounds'
constants are written in compressed form (one per round, see compress());
the script checks that both forms give the same permutation.

    python nitroozk-stwo_b200/csrc/poseidon252_constants.py
"""
import hashlib
import os

P = 2 ** 251 + 17 * 2 ** 192 + 1
R = 2 ** 256
N_ROUNDS = 8 + 83


def limbs(x):
    return ["0x%08xu" % ((x >> (32 * i)) & 0xFFFFFFFF) for i in range(8)]


def mont(x):
    return (x * R) % P


def felt_line(x):
    return "  {{" + ", ".join(limbs(x)) + "}}"


def limbs64(x):
    return "{" + ", ".join("0x%016xull" % ((x >> (64 * i)) & 0xFFFFFFFFFFFFFFFF) for i in range(4)) + "}"


MDS = [[3, 1, 1], [1, -1, 1], [1, 1, -2]]


def mds(v):
    return [sum(MDS[i][j] * v[j] for j in range(3)) % P for i in range(3)]


def permute_plain(s, rcs):
    s = list(s)
    for r in range(N_ROUNDS):
        s = [(x + rcs[3 * r + j]) % P for j, x in enumerate(s)]
        if r < 4 or r >= 4 + 83:
            s = [pow(x, 3, P) for x in s]
        else:
            s[2] = pow(s[2], 3, P)
        s = mds(s)
    return s


def compress(rcs):
    """Partial rounds with one constant each: in a partial round only s2 goes
    through the S-box, so the constants of s0 and s1 can be pushed through the
    MDS into the next round (MDS(x + (e0, e1, 0)) = MDS(x) + MDS((e0, e1,
    0))). Returns the 8 full rounds' constants (the first after the partial
    rounds absorbs what is still pending) and one constant per partial round."""
    full = [[rcs[3 * r + j] for j in range(3)] for r in list(range(4)) + list(range(87, 91))]
    part = []
    d = [0, 0, 0]
    for k in range(83):
        r = 4 + k
        e = [(d[j] + rcs[3 * r + j]) % P for j in range(3)]
        part.append(e[2])
        d = mds([e[0], e[1], 0])
    full[4] = [(full[4][j] + d[j]) % P for j in range(3)]
    return full, part


def permute_compressed(s, full, part):
    s = list(s)
    for r in range(4):
        s = mds([pow((x + full[r][j]) % P, 3, P) for j, x in enumerate(s)])
    for k in range(83):
        s[2] = pow((s[2] + part[k]) % P, 3, P)
        s = mds(s)
    for r in range(4, 8):
        s = mds([pow((x + full[r][j]) % P, 3, P) for j, x in enumerate(s)])
    return s


def main():
    rcs = []
    for r in range(N_ROUNDS):
        for j in range(3):
            rcs.append(int.from_bytes(hashlib.sha256(b"Hades%d" % (3 * r + j)).digest(), "big") % P)
    full, part = compress(rcs)
    for seed in range(4):  # the two forms are the same permutation
        st = [(seed * 1000003 + 7 * j + 1) ** 5 % P for j in range(3)]
        assert permute_plain(st, rcs) == permute_compressed(st, full, part)
    s2 = [row[2] for row in full[:4]] + part + [row[2] for row in full[4:]]  # s2's constant, by round
    s2_next = s2[1:] + [0]
    lines = [
        "// Generated by poseidon252_constants.py (do not edit): Starknet Poseidon",
        "// constants, Montgomery form (R = 2^256), 8 little-endian 32-bit limbs.",
        "__constant__ Felt P252_R2 = {{" + ", ".join(limbs((R * R) % P)) + "}};  // R^2 mod p",
        "__constant__ Felt P252_ONE = {{" + ", ".join(limbs(mont(1))) + "}};",
        "__constant__ Felt P252_TWO = {{" + ", ".join(limbs(mont(2))) + "}};",
        "// the 8 full rounds (4 before, 4 after the partial rounds), 3 constants each",
        "__constant__ Felt P252_FULL_RC[24] = {",
        ",\n".join(felt_line(mont(c)) for row in full for c in row),
        "};",
        "// what the MDS of round r adds to s2: the next round's constant plus 10p (10p alone after the last)",
        "__constant__ Felt P252_S2_NEXT[91] = {",
        ",\n".join(felt_line(mont(c) + 10 * P) for c in s2_next),
        "};",
        "",
    ]
    here = os.path.dirname(os.path.abspath(__file__))
    dst = os.path.join(here, "poseidon252_constants.inc")
    with open(dst, "w") as f:
        f.write("\n".join(lines))
    print("wrote", dst)
    host = [
        "// Generated by poseidon252_constants.py (do not edit): Starknet Poseidon",
        "// constants, Montgomery form (R = 2^256), 4 little-endian 64-bit limbs.",
        "static const uint64_t P252H_R2[4] = " + limbs64((R * R) % P) + ";  // R^2 mod p",
        "static const uint64_t P252H_ONE[4] = " + limbs64(mont(1)) + ";",
        "// the 8 full rounds (4 before, 4 after the partial rounds), 3 constants each",
        "static const uint64_t P252H_FULL_RC[24][4] = {",
        ",\n".join("  " + limbs64(mont(c)) for row in full for c in row),
        "};",
        "// one constant per partial round, added to s2",
        "static const uint64_t P252H_PARTIAL_RC[83][4] = {",
        ",\n".join("  " + limbs64(mont(c)) for c in part),
        "};",
        "",
    ]
    dst = os.path.join(here, "poseidon252_constants_host.inc")
    with open(dst, "w") as f:
        f.write("\n".join(host))
    print("wrote", dst)


if __name__ == "__main__":
    main()
