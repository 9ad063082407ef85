"""Emit qspec_b200/csrc/hadk_masks.inc and qspec_b200/_hadk.py from tests/golden/had108.npy / had40.npy (the reference's
get_had108 / get_had40 matrices, third-party/QuaRot/quarot/functional/hadamard.py, exported by tests/golden/make_golden.py):
the Qwen2.5-14B variant's rotations. Bit k of word k >> 5 of mask[o] is set iff H[o][k] == -1."""
import os
import numpy as np

root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
out_c = ["// Generated by scripts/gen_hadk_masks.py -- do not edit.\n"]
out_py = ['"""Generated by scripts/gen_hadk_masks.py -- the +-1 Hadamard matrices get_had108 / get_had40 of the reference\n'
          '(third-party/QuaRot/quarot/functional/hadamard.py) as row bit-masks (bit k of word k >> 5 of NEG[K][o] set <=> H[o][k] == -1)."""\n'
          "import torch\n\nNEG = {\n"]
for K in (108, 40):
    h = np.load(os.path.join(root, "tests", "golden", f"had{K}.npy"))
    assert h.shape == (K, K) and set(np.unique(h)) == {-1, 1}
    W = (K + 31) // 32
    masks = [[sum(1 << (k & 31) for k in range(K) if h[o, k] < 0 and (k >> 5) == w) for w in range(W)] for o in range(K)]
    out_c.append(f"__constant__ uint32_t d_had{K}_neg[{K}][{W}] = {{\n")
    out_c.append(",\n".join("  {" + ", ".join(f"0x{m:08x}u" for m in row) + "}" for row in masks))
    out_c.append("\n};\n")
    # the same signs as fp32 multipliers for the FMA form of the mix, laid out for 128-bit constant loads: [k][group][G4] float4,
    # group g holds the outputs o = g * per .. g * per + per - 1 (per = 27 for had108: 4 groups; 20 for had40: 2 groups), padded to G4 * 4
    per, groups = (27, 4) if K == 108 else (20, 2)
    g4 = (per + 3) // 4
    out_c.append(f"// sign multipliers (+1 / -1; 0 = padding): d_had{K}_sign[k][g][q] = (H[g * {per} + 4 q + 0..3][k])\n")
    space = "__device__ const" if K == 108 else "__constant__"      # had108: 47 KB, copied into shared memory by the kernel
    out_c.append(f"{space} float4 d_had{K}_sign[{K}][{groups}][{g4}] = {{\n")
    rows = []
    for k in range(K):
        grp = []
        for g in range(groups):
            vals = [float(h[g * per + i, k]) if i < per else 0.0 for i in range(g4 * 4)]
            grp.append("{" + ", ".join("{" + ", ".join(f"{v:.0f}.f" for v in vals[4 * q: 4 * q + 4]) + "}" for q in range(g4)) + "}")
        rows.append("  {" + ", ".join(grp) + "}")
    out_c.append(",\n".join(rows))
    out_c.append("\n};\n")
    out_py.append(f"    {K}: [\n" + "".join("        [" + ", ".join(f"0x{m:08x}" for m in row) + "],\n" for row in masks) + "    ],\n")
out_py.append("}\n\n\ndef hadK(K: int) -> torch.Tensor:\n"
              "    rows = [[-1.0 if (m[k >> 5] >> (k & 31)) & 1 else 1.0 for k in range(K)] for m in NEG[K]]\n"
              "    return torch.tensor(rows, dtype=torch.float32)\n")
open(os.path.join(root, "qspec_b200", "csrc", "hadk_masks.inc"), "w").write("".join(out_c))
open(os.path.join(root, "qspec_b200", "_hadk.py"), "w").write("".join(out_py))
print("ok")
