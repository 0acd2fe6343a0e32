// Which operands of the invariant point attention core (ipa.cu) are bf16 and not fp32; set by csrc/host/dispatch.cpp.
#pragma once

enum IpaBf16 { IPA_BF16_WB = 1, IPA_BF16_BB = 2, IPA_BF16_GAMMA = 4, IPA_BF16_MASK = 8 };
