"""The build's look at the compiler's report: kernels that split their registers among warpgroups and get too few at launch."""
from beglin_b200.csrc import build

ENTRY = "ptxas info    : Compiling entry function '%s' for 'sm_100a'\nptxas info    : Function properties for %s\n    0 bytes stack frame\nptxas info    : Used %d registers, used 2 barriers\n"
PRODUCT = "_ZN2bg18gemm_f32_tc_kernelINS_6GtFormILi16ELi4ELi1ELi4ELi4ELi5ELi4ELi80ELi72ELi64ELi72EEELb0EEEv14CUtensorMap_stNS_8GtParamsE"
ATTENTION = "_ZN2bg23attention_f32_tc_kernelINS_10AttnParamsELi64EEEvT_"


def report(**used):
    names = {"product": PRODUCT, "attention": ATTENTION, "other": "_ZN2bg15gf_parts_kernelILb0EEEvNS_8GtParamsEPhi"}
    return "".join(ENTRY % (names[k], names[k], n) for k, n in used.items())


def test_registers_short():
    want = build._attention_registers()
    assert build.registers_short(report(other=8, product=80, attention=want), want) == []
    assert build.registers_short(report(product=72, other=8, attention=want), want) == [f"{PRODUCT}: 72 registers of 80"]
    assert build.registers_short(report(product=80, attention=want - 8), want) == [f"{ATTENTION}: {want - 8} registers of {want}"]
