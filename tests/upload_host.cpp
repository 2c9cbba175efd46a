// Host build of the upload's return rule (mhd_upload.h) against a fake pointer query.
#include "../beta1_b200/csrc/mhd_upload.h"

namespace
{
int g_unregistered = 0, g_asked = 0;
struct Fake
{
    static bool unregistered(const void *)
    {
        ++g_asked;
        return g_unregistered != 0;
    }
};
} // namespace

extern "C" int upload_rule(int unregistered, int reads_pageable)
{
    g_unregistered = unregistered;
    return upload_source_is_read<Fake>(nullptr, reads_pageable) ? 1 : 0;
}
