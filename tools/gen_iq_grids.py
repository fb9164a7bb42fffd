"""Generates the public ggml IQ codebook tables (iq2xxs / iq2xs / iq3xxs / iq2s / iq3s / iq1s grids, ksigns) as C headers from the
`gguf` python package installed in this image (gguf 0.19.0, gguf/quants.py; the reference has none of its own):

    python tools/gen_iq_grids.py      -> blazr_b200/csrc/iq_grids.h  (device + host-check builds)
                                         (oracle/quant_oracle.c includes the same file: oracle/Makefile -I../blazr_b200/csrc)
"""
import os

import numpy as np
from gguf import quants

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def table(name, arr, cols):
    rows = [", ".join(str(int(v)) for v in arr[i]) for i in range(arr.shape[0])]
    body = ",\n".join("    {" + r + "}" for r in rows)
    return f"IQ_TABLE_QUAL const uint8_t {name}[{arr.shape[0]}][{cols}] = {{\n{body}\n}};\n"


def main():
    out = ["// GENERATED by tools/gen_iq_grids.py from gguf 0.19.0 (gguf/quants.py): public ggml IQ codebooks.  Do not edit.",
           "#pragma once", "#include <stdint.h>", "#ifndef IQ_TABLE_QUAL", "#define IQ_TABLE_QUAL static", "#endif", ""]
    for cls, name in ((quants.IQ2_XXS, "iq2xxs_grid"), (quants.IQ2_XS, "iq2xs_grid"), (quants.IQ3_XXS, "iq3xxs_grid"),
                      (quants.IQ2_S, "iq2s_grid"), (quants.IQ3_S, "iq3s_grid")):
        cls.init_grid()
        g = cls.grid.reshape(cls.grid_shape).astype(np.uint8)
        out.append(table(name, g, cls.grid_shape[1]))
    quants.IQ1_S.init_grid()
    g1 = quants.IQ1_S.grid.reshape(quants.IQ1_S.grid_shape).astype(np.int8)   # values -1, 0, 1
    out.append(table("iq1s_grid", g1, 8).replace("const uint8_t iq1s_grid", "const int8_t iq1s_grid"))
    ks = np.frombuffer(quants.IQ2_XXS.ksigns, dtype=np.uint8)
    out.append("IQ_TABLE_QUAL const uint8_t iq_ksigns[128] = {" + ", ".join(str(int(v)) for v in ks) + "};\n")
    text = "\n".join(out)
    for rel in ("blazr_b200/csrc/iq_grids.h",):  # one copy: oracle/Makefile adds -I../blazr_b200/csrc
        open(os.path.join(ROOT, rel), "w").write(text)
        print("wrote", rel, len(text), "bytes")


if __name__ == "__main__":
    main()
